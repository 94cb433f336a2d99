// Symmetric recursive Green sweep for Dirichlet guides of up to 64 modes.
//
// With Dirichlet modes the slice matrix X_n = A_n - V_n - B Gss B is complex
// symmetric (A and B diagonal, V real symmetric, and Gss = inv(X_{n-1}) is
// symmetric in turn).  The kernel keeps it in the variables scaled by
// D = B^(1/2) (src/waveguide.f90:426-440 in them):
//   X' = D^-1 X D^-1 = A/B - D^-1 V D^-1 - G',   G' = D Gss D = inv(X'),
//   Q  = (D Gs1 D)^T:  Q_0 = G'_0,  Q_n = -Q_{n-1} G'_n,
// so a slice needs no product with B, and every matrix entry is of order 1.
//
// Why not FP64 elimination: FP64 is 1.7 FMA lanes per clock and SM here, so
// the 12 M^3 flops of a Gauss-Jordan sweep on [X | B Gs1] cost 49,000 warp
// instructions of 18 clocks per slice at M = 64 (0.9 M clocks), whatever the
// occupancy.  Instead, per slice:
//   1. X'^-1 in FP32 (Y0; block Gauss-Jordan on the 16 x 16 tiles that the
//      warps hold in registers), rounded to 26-bit fixed point;
//   2. its residual R = I - Y0 X' exactly enough (2^-58), on the FP16 tensor
//      cores with the balanced 9-bit digits of rg_ozaki.cuh, seven of them
//      for X' (with six, its rounding relative to the row's largest entry
//      doubled the error of t);
//   3. G' = (I + R + R^2 + ...) Y0: E_1 = R Y0, E_k+1 = R E_k, summed in
//      64-bit fixed point until ||R||^(k+1) is below 2^-55.  ||R|| is near
//      1e-5, so three terms do, and the digits kept in each follow from the
//      magnitudes;
//   4. Q on the tensor cores, all 26 digit pairs, rounded once.
// FP64 instructions are left in the potential's draw and projection, which
// two producer warps run one slice ahead of the others, and in the assembly
// of X'.  The residual makes the result as accurate as an FP64 inverse: the
// error of t against an extended-precision sweep is that of the elimination
// within 0.95 to 1.3 (7 to 64 modes, 40 to 300 slices; geometric mean 1.08).
// Measured, with the eigenvalues: 304 guides of 64 modes and 600 slices 607 ms
// before, 184 now; 500 of 37 modes and 150 slices 110 ms before, 41 now; one
// guide of 10 modes and 200 slices 8.2 ms before, 4.4 now.
//
// Layout: T = ceil(M/16) tiles a side, one warp per tile (ti, tj) in the
// accumulator layout of mma.m16n8k16, which for two n8 tiles is also the
// fragment layout of its A operand and, read as the transpose, of its B
// operand: digits go from registers to shared memory and back without a
// shuffle, and one set of planes serves both sides of a symmetric matrix.
// (Q is kept transposed so that it is only ever an A operand.)  Two plane
// regions of 12 x T^2 x 512 bytes are reused through the slice:
//   region A: X' -> R -> G';   region B: Y0 -> E_k -> Q.
// Q, G' and the scaling products w_i w_j stay with their owner lanes, in the
// CTA's workspace (L2).  At 33 to 48 modes two CTAs fit on an SM, at 49 to
// 64 one.
//
// If a pivot is too small against the unswept entries of its row (sym_tau),
// or the residual is not small, the item is flagged (kStatusNeedPivot), its
// index appended to a.flag_list, and it is recomputed by the pivoted kernel,
// which launch_sweep starts on that list.
#include "rg_device.cuh"
#include "rg_ozaki.cuh"

namespace rg {
namespace {

__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// Named barriers: the main warps, the producer warps, and the two buffers of
// projection coefficients (filled / free again).
constexpr int kBarMain = 1, kBarProd = 2, kBarFull = 3, kBarFree = 5;

// Fixed point: Y0 has 26 bits, the sum of the series 56, relative to the
// power of two of the row.
constexpr int kY0Bits = 26, kAccBits = 56;

// Pivots of the FP32 elimination come in natural order, and the residual of
// its result is checked, so they may be this much smaller against their row
// than sym_tau asks of a pivot that was searched for.
constexpr double kNaturalTau = 0.1;

template <int T>
struct SymCfg {
  static constexpr int MP = 16 * T;                // padded modes
  static constexpr int NE = T == 4 ? 8 : 4;        // complex entries per lane: a whole tile, or its column half
  static constexpr int NHALF = 8 / NE;             // warps per tile
  static constexpr int NCW = T * NHALF;            // warps that share a row
  static constexpr int NMAIN = 32 * T * T * NHALF;
  // Producer threads.  Registers are handed out to four warps at a time.
  static constexpr int PROD = T == 4 ? 128 : 64;
  static constexpr int NT = NMAIN + PROD;
  static constexpr int MINB = T == 1 ? 4 : T == 2 ? 2 : 1;  // CTAs per SM
  static constexpr int PL = T * T * 32;            // uint4 of one digit plane
  static constexpr int LDW = MP + 1;
  static constexpr size_t bytes() {
    return sizeof(uint4) * 24 * PL + sizeof(double) * (2 * (2 * MP + 2) + PROD) + sizeof(unsigned long long) * 2 +
           sizeof(unsigned) * 32 + sizeof(int) * 3 * NCW * MP;
  }
};

// Workspace of one CTA in double2: generator states (ny x 4 uint64), the
// potential row, then Q, G' and w_i w_j by warp, element and lane.
inline int64_t sym_stride(int T, int max_ny) {
  return (2 * (int64_t)max_ny + (max_ny + 1) / 2 + 3 * (int64_t)T * T * 256 + 15) & ~(int64_t)15;
}

// Bits of |x| of a float, 0 for NaN (so that NaN never wins a pivot search).
__device__ __forceinline__ unsigned fkey(float2 x) {
  const unsigned a = __float_as_uint(x.x) & 0x7fffffffu, b = __float_as_uint(x.y) & 0x7fffffffu;
  const unsigned m = a > b ? a : b;
  return m > 0x7f800000u ? 0u : m;
}

// x rounded towards zero to FP32, in integer instructions (a conversion
// instruction runs on the FP64 pipe).
__device__ __forceinline__ float to_f32(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const unsigned hi = (unsigned)(b >> 32);
  const int e = (int)((hi >> 20) & 0x7ff) - 896;
  const unsigned s = hi & 0x80000000u;
  if (e <= 0) return __uint_as_float(s);
  if (e >= 255) return __uint_as_float(s | (e == 1151 && (b << 12) ? 0x7fc00000u : 0x7f800000u));
  return __uint_as_float(s | ((unsigned)e << 23) | (unsigned)((b >> 29) & 0x7fffffu));
}

__device__ __forceinline__ float2 fcmul(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
// a b + c on both halves (one instruction)
__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) {
  unsigned long long x, y, z, r;
  memcpy(&x, &a, 8);
  memcpy(&y, &b, 8);
  memcpy(&z, &c, 8);
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(x), "l"(y), "l"(z));
  float2 o;
  memcpy(&o, &r, 8);
  return o;
}

// Entry k of a lane: row g + erow(k), column 2 t + ecol(k) (plus 8 in the
// second half of a split tile), with g = lane / 4, t = lane % 4.
__device__ __forceinline__ constexpr int erow(int k) { return 8 * ((k >> 1) & 1); }
__device__ __forceinline__ constexpr int ecol(int k) { return (k & 1) + 8 * (k >> 2); }

// A published FP32 tile: rows of 18 complex, so that the eight rows a warp
// reads at once lie in different banks.
constexpr int kTileLd = 18, kTileF2 = 16 * kTileLd;

// m -= A B over the 16 columns of A, for a lane's entries (rows g, g + 8;
// columns lc, lc + 1 and, for a whole tile, 8 further on).  A product f s is
// (-f.x, -f.x) (s.x, s.y) + (f.y, -f.y) (s.y, s.x): two packed FMAs.
template <int NE>
__device__ __forceinline__ void tile_fms(float2* m, const float2* A, const float2* B, int g, int lc) {
#pragma unroll 4
  for (int k = 0; k < 16; ++k) {
    const float2 f0 = A[g * kTileLd + k], f1 = A[(g + 8) * kTileLd + k];
    const float2 f0r = make_float2(-f0.x, -f0.x), f0i = make_float2(f0.y, -f0.y);
    const float2 f1r = make_float2(-f1.x, -f1.x), f1i = make_float2(f1.y, -f1.y);
#pragma unroll
    for (int q = 0; q < NE; q += 4) {
      const float4 u = *reinterpret_cast<const float4*>(B + k * kTileLd + lc + 2 * q);
      const float2 s0 = make_float2(u.x, u.y), s1 = make_float2(u.z, u.w);
      const float2 t0 = make_float2(s0.y, s0.x), t1 = make_float2(s1.y, s1.x);
      m[q] = ffma2(f0i, t0, ffma2(f0r, s0, m[q]));
      m[q + 1] = ffma2(f0i, t1, ffma2(f0r, s1, m[q + 1]));
      m[q + 2] = ffma2(f1i, t0, ffma2(f1r, s0, m[q + 2]));
      m[q + 3] = ffma2(f1i, t1, ffma2(f1r, s1, m[q + 3]));
    }
  }
}

// The leading n x n part of the complex symmetric tile at P inverted in place
// by one warp (the rest stays zero): symmetric Gauss-Jordan, pivots in natural
// order.  After sweeping 0..p-1 the in-place matrix satisfies M[i][j] =
// +-M[j][i], minus when exactly one of i, j is swept.  Sweeping p with z =
// M[p][p], d = 1/z, r_j = M[p][j] and g_i = M[i][p]:
//   M[i][j] -= g_i d r_j (i, j != p),  M[p][j] = d r_j,  M[i][p] = -g_i d,
//   M[p][p] = d;
// the pivot row and column take the same form, M[i][j] -= f_i s_j with f_p =
// 1 - d (else g_i d) and s_p = z + 1 (else r_j).  Row p passes through the
// tile's own row in shared memory.  Returns true when a pivot falls below tau
// times the largest unswept entry of its row.
__device__ __forceinline__ bool invert_tile(float2* P, int n, float tau, int lane) {
  const int g = lane >> 2, c = 2 * (lane & 3);
  float2 m[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) m[q] = P[(g + erow(q)) * kTileLd + c + ecol(q)];
  bool small_pivot = false;
#pragma unroll
  for (int hh = 0; hh < 2; ++hh) {
#pragma unroll 1
    for (int p = 8 * hh; p < min(n, 8 * hh + 8); ++p) {
      float2* rb = P + p * kTileLd;
      if (g == (p & 7)) {
#pragma unroll
        for (int q = 0; q < 8; q += 4) {
          const float2 u0 = m[q + 2 * hh], u1 = m[q + 2 * hh + 1];
          *reinterpret_cast<float4*>(rb + c + 2 * q) = make_float4(u0.x, u0.y, u1.x, u1.y);
        }
      }
      __syncwarp();
      const float2 z = rb[p];
      const float2 u0 = rb[g], u1 = rb[g + 8];
      const float4 v0 = *reinterpret_cast<const float4*>(rb + c), v1 = *reinterpret_cast<const float4*>(rb + c + 8);
      const float rden = __fdividef(1.0f, fmaf(z.x, z.x, z.y * z.y));
      const float2 d = make_float2(z.x * rden, -z.y * rden), dn = make_float2(-d.x, -d.y);
      const float2 fp = make_float2(1.0f - d.x, -d.y);
      float2 f0 = fcmul(u0, g < p ? dn : d), f1 = fcmul(u1, g + 8 < p ? dn : d);
      if (g == p) f0 = fp;
      if (g + 8 == p) f1 = fp;
      const float zk = fmaxf(fabsf(z.x), fabsf(z.y));
      const float2 f0r = make_float2(-f0.x, -f0.x), f0i = make_float2(f0.y, -f0.y);
      const float2 f1r = make_float2(-f1.x, -f1.x), f1i = make_float2(f1.y, -f1.y);
#pragma unroll
      for (int q = 0; q < 8; q += 4) {
        const float4 u = q ? v1 : v0;
        const int cq = c + 2 * q;
        if (cq > p && zk < tau * fmaxf(fabsf(u.x), fabsf(u.y))) small_pivot = true;
        if (cq + 1 > p && zk < tau * fmaxf(fabsf(u.z), fabsf(u.w))) small_pivot = true;
        const float2 s0 = make_float2(cq == p ? u.x + 1.0f : u.x, u.y);
        const float2 s1 = make_float2(cq + 1 == p ? u.z + 1.0f : u.z, u.w);
        const float2 t0 = make_float2(s0.y, s0.x), t1 = make_float2(s1.y, s1.x);
        m[q] = ffma2(f0i, t0, ffma2(f0r, s0, m[q]));
        m[q + 1] = ffma2(f0i, t1, ffma2(f0r, s1, m[q + 1]));
        m[q + 2] = ffma2(f1i, t0, ffma2(f1r, s0, m[q + 2]));
        m[q + 3] = ffma2(f1i, t1, ffma2(f1r, s1, m[q + 3]));
      }
      __syncwarp();
    }
  }
#pragma unroll
  for (int q = 0; q < 8; ++q) P[(g + erow(q)) * kTileLd + c + ecol(q)] = m[q];
  return __any_sync(0xffffffffu, small_pivot);
}

template <int T>
__global__ void __launch_bounds__(SymCfg<T>::NT, SymCfg<T>::MINB) sweep_sym_kernel(SweepArgs a) {
  using Cf = SymCfg<T>;
  constexpr int MP = Cf::MP, NMAIN = Cf::NMAIN, NT = Cf::NT, PL = Cf::PL, LDW = Cf::LDW, kProd = Cf::PROD;
  constexpr int NE = Cf::NE, NV = 2 * NE, NHALF = Cf::NHALF, NCW = Cf::NCW;
  extern __shared__ uint4 smem[];
  uint4* regA = smem;                          // 12 planes
  uint4* regB = smem + 12 * PL;                // 12 planes
  double* cc = (double*)(smem + 24 * PL);      // [2][2 MP + 2] projection coefficients
  double* part = cc + 2 * (2 * MP + 2);        // [kProd] partial projections
  unsigned long long* rsum = (unsigned long long*)(part + kProd);  // [2] sum of squares of the residual
  unsigned* red = (unsigned*)(rsum + 2);       // [32] maxima of a slice
  int* exX = (int*)(red + 32);                 // [NCW][MP] row exponents by warp column: X',
  int* exY = exX + NCW * MP;                   // Y0,
  int* exQ = exY + NCW * MP;                   // Q
  __shared__ int s_r;
  __shared__ volatile int s_status, s_abort[2];
  __shared__ WgDesc wd;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool main_thread = tid < NMAIN;
  const int g = lane >> 2, t4 = lane & 3;
  const int tile = warp / NHALF, half = NHALF == 2 ? warp & 1 : 0;
  const int ti = tile / T, tj = tile % T;
  const int r0 = ti * 16 + g, c0 = tj * 16 + 2 * t4 + 8 * half;
  double2* ws = a.work + (int64_t)blockIdx.x * a.work_stride;
  uint64_t* gen = (uint64_t*)ws;               // [max_ny][4]
  double* urow = (double*)(ws + 2 * (int64_t)a.max_ny);  // [max_ny] potential row
  double2* Qs = ws + 2 * (int64_t)a.max_ny + (a.max_ny + 1) / 2 + (main_thread ? warp * 32 * NE + lane : 0);
  double2* Gs = Qs + T * T * 256;              // entry k of this lane at [32 k]
  double2* Ww = Gs + T * T * 256;
  // This lane's place in the planes: its tile, and the word pairs of its tile
  // row (as A) and tile column (as B), in bytes.
  constexpr int kPlane = 16 * PL;
  const int odd = (lane >> 3) & 1;
  const int own = tile * 32 + lane;
  const int offA0 = ti * T * 512 + lane * 16 + 8 * odd, offA1 = ti * T * 512 + lane * 16 + 8 * (1 - odd);
  const int offB = tj * T * 512 + lane * 16;
  const char* bA = (const char*)regA;
  const char* bB = (const char*)regB;
  const bool draw = (a.upot == nullptr);
  const bool tmat = (a.mode == kModeTmat);
  const bool refl = (a.mode == kModeRefl);
  const float tau = (float)fmin(kNaturalTau * a.sym_tau, 3e38);

  auto mbar = [&]() {
    if (NMAIN == 32) __syncwarp();
    else bar_sync(kBarMain, NMAIN);
  };

  for (;;) {
    if (tid == 0) {
      s_r = atomicAdd(a.work_counter, 1);
      if (s_r < a.nreal) wd = a.wgs[a.item_wg ? a.item_wg[s_r] : 0];
    }
    __syncthreads();
    const int r = s_r;
    if (r >= a.nreal) break;
    const int M = wd.M, ny = wd.ny, nx = wd.nx;
    const bool per = wd.periodic != 0;  // X is Hermitian there, not symmetric
    if (tid == 0) {
      s_status = per ? kStatusNeedPivot : RG_OK;
      s_abort[0] = s_abort[1] = 0;
    }
    __syncthreads();

    if (per) {
      // handed to the pivoted kernel below
    } else if (!main_thread) {
      // Producers: the potential row of slice n and its projection
      // cc[d] = sum_j costab[j][d] U_j, one slice ahead.  The transverse grid
      // is symmetric (y_{ny-1-j} = 1 - y_j) and cos(pi d (1 - y)) =
      // (-1)^d cos(pi d y), so the points pair up as sums (even d) and
      // differences (odd d) over half the points.
      const int pt = tid - NMAIN;
      const double* U = draw ? nullptr : a.upot + (int64_t)r * a.pot_rstride;
      if (draw)
        for (int j = pt; j < ny; j += kProd) {
          const Xoshiro st = jump_state(seeded_state(a.seeds[r]), wd.jumppoly + 4 * (int64_t)j);
          gen[4 * j + 0] = st.s0;
          gen[4 * j + 1] = st.s1;
          gen[4 * j + 2] = st.s2;
          gen[4 * j + 3] = st.s3;
        }
      const int h = ny >> 1, nd = 2 * M + 1;
      for (int n = 0; n < nx; ++n) {
        const int b = n & 1;
        if (n >= 2) bar_sync(kBarFree + b, NT);
        const int id = (refl ? nx - 1 - n : n) - wd.nxfree;
        if (id >= 0 && id < wd.nxdiso && !s_abort[b]) {
          for (int j = pt; j < ny; j += kProd) {
            double u;
            if (draw) {
              Xoshiro st{gen[4 * j], gen[4 * j + 1], gen[4 * j + 2], gen[4 * j + 3]};
              u = scaled_normal(wd.stdu, st);
              gen[4 * j + 0] = st.s0;
              gen[4 * j + 1] = st.s1;
              gen[4 * j + 2] = st.s2;
              gen[4 * j + 3] = st.s3;
            } else {
              u = U[(int64_t)id * a.pot_xstride + (int64_t)j * a.pot_ystride];
            }
            urow[j] = u;
          }
          bar_sync(kBarProd, kProd);
          for (int j = pt; j < h; j += kProd) {
            const double u0 = urow[j], u1 = urow[ny - 1 - j];
            urow[j] = u0 + u1;
            urow[ny - 1 - j] = u0 - u1;
          }
          bar_sync(kBarProd, kProd);
          double* co = cc + b * (2 * MP + 2);
          auto dot = [&](int d, int j, int j1, bool mid) {  // sum over [j, j1) and the middle point
            const double* ct = wd.costab + d;
            const double* up = (d & 1) ? urow + (ny - 1) : urow;
            const int us = (d & 1) ? -1 : 1;
            double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
            for (; j + 4 <= j1; j += 4) {
              s0 = fma(ct[(int64_t)(j + 0) * nd], up[us * (j + 0)], s0);
              s1 = fma(ct[(int64_t)(j + 1) * nd], up[us * (j + 1)], s1);
              s2 = fma(ct[(int64_t)(j + 2) * nd], up[us * (j + 2)], s2);
              s3 = fma(ct[(int64_t)(j + 3) * nd], up[us * (j + 3)], s3);
            }
            for (; j < j1; ++j) s0 = fma(ct[(int64_t)j * nd], up[us * j], s0);
            if (mid && (ny & 1)) s1 = fma(ct[(int64_t)h * nd], urow[h], s1);
            return (s0 + s1) + (s2 + s3);
          };
          if (kProd > 32 && 2 * nd <= kProd) {  // several threads share a coefficient
            const int nseg = kProd / nd, seg = pt / nd, d = pt % nd;
            if (seg < nseg) part[pt] = dot(d, seg * h / nseg, (seg + 1) * h / nseg, seg == nseg - 1);
            bar_sync(kBarProd, kProd);
            if (pt < nd) {
              double s = part[pt];
              for (int k = 1; k < nseg; ++k) s += part[k * nd + pt];
              co[pt] = s;
            }
          } else {
            // the coefficients beyond a multiple of kProd take a round of
            // their own, or a warp each with a shuffle reduction
            const int rem = nd % kProd;
            const bool byw = rem * ((h + 31) / 32 + 5) < 2 * h;
            const int full = byw ? nd - rem : nd;
            for (int d = pt; d < full; d += kProd) co[d] = dot(d, 0, h, true);
            for (int d = full + (pt >> 5); d < nd; d += kProd / 32) {
              const double* ct = wd.costab + d;
              const double* up = (d & 1) ? urow + (ny - 1) : urow;
              const int us = (d & 1) ? -1 : 1;
              double s0 = 0.0;
              for (int j = lane; j < h; j += 32) s0 = fma(ct[(int64_t)j * nd], up[us * j], s0);
              if ((ny & 1) && lane == 0) s0 = fma(ct[(int64_t)h * nd], urow[h], s0);
#pragma unroll
              for (int off = 16; off; off >>= 1) s0 += __shfl_xor_sync(0xffffffffu, s0, off);
              if (lane == 0) co[d] = s0;
            }
          }
          bar_sync(kBarProd, kProd);  // urow is read before the next slice draws into it
        }
        bar_arrive(kBarFull + b, NT);
      }
    } else {
      // Scaling products w_i w_j of this lane's elements.
      bool real_w = true;
#pragma unroll
      for (int k = 0; k < NE; ++k) {
        const int i = r0 + erow(k), j = c0 + ecol(k);
        double2 v = make_double2(0.0, 0.0);
        if (i < M && j < M) v = cmul(wd.wsc[i], wd.wsc[j]);
        Ww[32 * k] = v;
        real_w = real_w && v.y == 0.0;
      }
      real_w = __all_sync(0xffffffffu, real_w);
      bool aborted = false;
      for (int n = 0; n < nx; ++n) {
        const int b = n & 1;
        bar_sync(kBarFull + b, NT);
        double2 x[NE];
        if (!aborted) {
          // 1. X' = A/B - w V w - G' (zero outside M x M).
          const int id = (refl ? nx - 1 - n : n) - wd.nxfree;
          const bool dis = (id >= 0 && id < wd.nxdiso), edge = (n == 0 || n == nx - 1);
          const double* co = cc + b * (2 * MP + 2);
#pragma unroll
          for (int k = 0; k < NE; ++k) {
            const int i = r0 + erow(k), j = c0 + ecol(k);
            double2 v = make_double2(0.0, 0.0);
            if (i < M && j < M) {
              if (n > 0) {
                v = Gs[32 * k];
                v = make_double2(-v.x, -v.y);
              }
              if (i == j) {
                const double2 d = edge ? wd.aw_edge[i] : wd.aw_bulk[i];
                v = make_double2(v.x + d.x, v.y + d.y);
              }
              if (dis) {
                const double vij = co[i > j ? i - j : j - i] - co[i + j + 2];
                const double2 w = Ww[32 * k];
                v.x = fma(-w.x, vij, v.x);
                if (!real_w) v.y = fma(-w.y, vij, v.y);
              }
              if (i == j) {  // the rest of A/B beyond FP64
                const double2 d = edge ? wd.aw_edge[M + i] : wd.aw_bulk[M + i];
                v = make_double2(v.x + d.x, v.y + d.y);
              }
            }
            x[k] = v;
          }
        }
        if (n <= nx - 3) {
          if (tid == 0) s_abort[b] = aborted ? 1 : 0;
          bar_arrive(kBarFree + b, NT);
        }
        if (aborted) continue;

        // Row exponents over the warps of a row, then the planes of X'.
        float2 m[NE];
        uint32_t x7[NE];  // the seventh digit of X'
        {
          int e0 = oz::kNoExp, e1 = oz::kNoExp;
#pragma unroll
          for (int k = 0; k < NE; ++k) {
            if (erow(k)) e1 = max(e1, oz::fexp2(x[k]));
            else e0 = max(e0, oz::fexp2(x[k]));
          }
          oz::put_row_exps(exX + (tj * NHALF + half) * MP, ti, lane, e0, e1);
          mbar();
          if (tid < 32) red[tid] = 0;
          if (tid == 0) rsum[0] = 0;
          e0 = oz::row_exp<NCW>(exX, MP, r0);
          e1 = oz::row_exp<NCW>(exX, MP, r0 + 8);
          long long fx[NV];
#pragma unroll
          for (int k = 0; k < NE; ++k) {
            const int e = erow(k) ? e1 : e0;
            fx[k] = oz::sfixed62(x[k].x, e);
            fx[NE + k] = oz::sfixed62(x[k].y, e);
            m[k] = make_float2(to_f32(x[k].x), to_f32(x[k].y));
          }
          oz::put_planes<62, NE>(fx, 6, regA + own, PL, 6, half, 0, x7);
        }

        // 2. Y0: block Gauss-Jordan in FP32 on the tiles in registers, pivot
        //    tiles in natural order.  Step t: P = M_tt^-1 by one warp
        //    (invert_tile), then
        //      M_tj <- P M_tj,  M_ij <- M_ij - M_it M_tj  (new M_tj),
        //      M_it <- -M_it P,  M_tt <- P       (i, j != t),
        //    16-term sums at full FMA rate between four barriers.  Scalar
        //    steps over the whole matrix took 1,000 clocks each at T = 4 (64
        //    of them: two barriers, or an mbarrier, and a chain of loads and
        //    FMAs a step); searching the largest diagonal entry would halve
        //    the residual, which the series absorbs as well.
        float2* tbuf = (float2*)regB;               // published tiles, kTileF2 apart:
        float2* Pt = tbuf;                          //   M_tt, then P
        float2* Ct = tbuf + kTileF2;                //   [T] column tiles M_it (T > 1)
        float2* Rt = Ct + T * kTileF2;              //   [T] row tiles M_tj
        float2* St = Rt + T * kTileF2;              //   [T] P M_tj
        const int lc = 2 * t4 + 8 * half;           // this lane's first column inside the tile
        auto put_tile = [&](float2* dst) {
#pragma unroll
          for (int q = 0; q < NE; q += 2)
            *reinterpret_cast<float4*>(dst + (g + erow(q)) * kTileLd + lc + (q & 4 ? 8 : 0)) =
                make_float4(m[q].x, m[q].y, m[q + 1].x, m[q + 1].y);
        };
        bool small_pivot = false;
#pragma unroll 1
        for (int t = 0; t < T; ++t) {
          if (16 * t >= M) break;
          if (ti == t && tj == t) put_tile(Pt);
          if (T > 1) {
            if (tj == t && ti != t) put_tile(Ct + ti * kTileF2);
            if (ti == t && tj != t) put_tile(Rt + tj * kTileF2);
          }
          mbar();
          if (ti == t && tj == t && half == 0) small_pivot |= invert_tile(Pt, min(16, M - 16 * t), tau, lane);
          mbar();
          if (ti == t && tj == t) {
#pragma unroll
            for (int q = 0; q < NE; ++q) m[q] = Pt[(g + erow(q)) * kTileLd + lc + ecol(q)];
          } else if (T > 1 && (ti == t || tj == t)) {
#pragma unroll
            for (int q = 0; q < NE; ++q) m[q] = make_float2(0.0f, 0.0f);
            if (ti == t) tile_fms<NE>(m, Pt, Rt + tj * kTileF2, g, lc);
            else tile_fms<NE>(m, Ct + ti * kTileF2, Pt, g, lc);
            if (ti == t) {
#pragma unroll
              for (int q = 0; q < NE; ++q) m[q] = make_float2(-m[q].x, -m[q].y);
              put_tile(St + tj * kTileF2);
            }
          }
          if (T > 1) {
            mbar();
            if (ti != t && tj != t) tile_fms<NE>(m, Ct + ti * kTileF2, St + tj * kTileF2, g, lc);
            mbar();
          }
        }
        if (small_pivot) s_status = kStatusNeedPivot;
        // Y0 made exactly symmetric (the entries below the diagonal from
        // above it), so that its planes serve as both operands.
        float2* sy = (float2*)(regB + 6 * PL);  // [MP][LDW]
#pragma unroll
        for (int k = 0; k < NE; ++k) sy[(r0 + erow(k)) * LDW + c0 + ecol(k)] = m[k];
        mbar();
        aborted = s_status == kStatusNeedPivot;
        if (aborted) continue;
#pragma unroll
        for (int k = 0; k < NE; ++k) {
          const int i = r0 + erow(k), j = c0 + ecol(k);
          if (i > j) m[k] = sy[j * LDW + i];
        }
        int ey0, ey1;
        long long acc[NV];  // the sum of the series, kAccBits of the row's power of two
        {
          unsigned k0 = 0, k1 = 0;
#pragma unroll
          for (int k = 0; k < NE; ++k) {
            if (erow(k)) k1 = max(k1, fkey(m[k]));
            else k0 = max(k0, fkey(m[k]));
          }
          oz::put_row_exps(exY + (tj * NHALF + half) * MP, ti, lane, k0 ? (int)(k0 >> 23) - 126 : oz::kNoExp,
                           k1 ? (int)(k1 >> 23) - 126 : oz::kNoExp);
          mbar();
          ey0 = oz::row_exp<NCW>(exY, MP, r0);
          ey1 = oz::row_exp<NCW>(exY, MP, r0 + 8);
          // 2^(26 - e) as a float (e within +-100; anything else is flagged by the residual)
          const float s0 = __uint_as_float((unsigned)(127 + kY0Bits - max(-100, min(100, ey0))) << 23);
          const float s1 = __uint_as_float((unsigned)(127 + kY0Bits - max(-100, min(100, ey1))) << 23);
#pragma unroll
          for (int k = 0; k < NE; ++k) {
            const float f = erow(k) ? s1 : s0;
            acc[k] = __float2int_rn(m[k].x * f);
            acc[NE + k] = __float2int_rn(m[k].y * f);
          }
          oz::put_planes<kY0Bits, NE>(acc, 3, regB + own, PL, 3, half);
          oz::put_words<NE>(x7, regB + 6 * PL + own, odd, half);
          oz::put_words<NE>(x7 + NE / 2, regB + 7 * PL + own, odd, half);
#pragma unroll
          for (int k = 0; k < NV; ++k) acc[k] *= 1LL << (kAccBits - kY0Bits);
        }
        mbar();

        // 3. R = I - Y0 X' at 2^-62, its largest entry and Frobenius norm.
        long long v[NV];
        unsigned mx = 0;
        unsigned long long sq = 0;
#pragma unroll
        for (int h = 0; h < NE / 4; ++h) {
          long long hi[8], lo[8];
          oz::half_product<T, 3, 7, oz::kLmax>(bB + offA0, bB + offA1, 3 * kPlane, bA + offB + 8 * (odd ^ (half | h)),
                                               6 * kPlane, kPlane, hi, lo,
                                               bB + 6 * kPlane + offB + 8 * (odd ^ (half | h)));
#pragma unroll
          for (int w = 0; w < 8; ++w) {
            const int k = 4 * h + (w & 3);
            const int i = r0 + erow(k), j = c0 + ecol(k);
            const int e = (erow(k) ? ey1 : ey0) + oz::row_exp<NCW>(exX, MP, j);
            long long y = 0;
            if (i < M && j < M) {
              const int up = 35 - e;  // |Y0 X'| < 2, or the inverse is useless
              const long long top = hi[w] + (lo[w] >> 36);
              const bool fits = up >= 62 || (up >= 0 ? (top >> up) == 0 || (top >> up) == -1 : top == 0);
              y = (w < 4 && i == j ? 1LL << 62 : 0) - oz::fix_shift(hi[w], lo[w], 28 + e);
              const unsigned long long av = (unsigned long long)(y < 0 ? -y : y);
              mx = max(mx, fits ? (unsigned)(av >> 32) : ~0u);
              const unsigned long long q = min(av >> 36, 1ULL << 26);
              sq += q * q;
            }
            v[(w < 4 ? 0 : NE) + k] = y;
          }
        }
        mx = __reduce_max_sync(0xffffffffu, mx);
#pragma unroll
        for (int off = 16; off; off >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, off);
        if (lane == 0) {
          atomicMax(red, mx);
          atomicAdd(rsum, sq);
        }
        mbar();
        const int er = 2 - __clz((int)red[0]);  // |R| < 2^er (at least 2^-30)
        const float rn = sqrtf((float)rsum[0]) * 0x1p-26f + (float)M * 0x1p-25f;
        if (!(rn < 0.125f) || er > -2) {
          aborted = true;
          if (tid == 0) s_status = kStatusNeedPivot;
          continue;
        }
        // Levels of a product of R with a matrix below 2^s of its row's power
        // of two: the dropped ones stay below 2^-57 of it.
        auto levels = [&](int s) { return max(0, min(oz::kLmax, (62 + er + s + 8) / 9 - 1)); };
        // E_1 = R Y0, E_k+1 = R E_k; the sum starts from Y0.
        int lm = levels(0);
        oz::put_planes<53, NE>(v, 6, regA + own, PL, 6, half, 9 + er);
        mbar();
        float rk = rn;  // ||R||^k of the term just formed
        int sk = 0;     // the B operand's entries are below 2^(e_i + sk)
        for (int term = 1;; ++term) {
          mx = 0;
#pragma unroll
          for (int h = 0; h < NE / 4; ++h) {
            long long hi[8], lo[8];
            const char* b = bB + offB + 8 * (odd ^ (half | h));
            if (term == 1) {
              if (lm <= 4) oz::half_product<T, 5, 3, 4>(bA + offA0, bA + offA1, 6 * kPlane, b, 3 * kPlane, kPlane, hi, lo);
              else oz::half_product<T, 6, 3, 6>(bA + offA0, bA + offA1, 6 * kPlane, b, 3 * kPlane, kPlane, hi, lo);
            } else if (lm == 0) {
              oz::half_product<T, 1, 1, 0>(bA + offA0, bA + offA1, 6 * kPlane, b, 6 * kPlane, kPlane, hi, lo);
            } else if (lm <= 2) {
              oz::half_product<T, 3, 3, 2>(bA + offA0, bA + offA1, 6 * kPlane, b, 6 * kPlane, kPlane, hi, lo);
            } else {
              oz::half_product<T, 6, 6, 6>(bA + offA0, bA + offA1, 6 * kPlane, b, 6 * kPlane, kPlane, hi, lo);
            }
#pragma unroll
            for (int w = 0; w < 8; ++w) {
              const int k = 4 * h + (w & 3);
              const int e = oz::row_exp<NCW>(exY, MP, c0 + ecol(k)) - (erow(k) ? ey1 : ey0);
              // rounded: truncating, a bias of 2^-57 in every entry, is an
              // error of M 2^-57 in norm that adds up from slice to slice
              const long long y = (oz::fix_shift(hi[w], lo[w], kAccBits - 33 + er + sk + e) + 1) >> 1;
              const int q = (w < 4 ? 0 : NE) + k;
              acc[q] += y;
              v[q] = y;
              mx = max(mx, (unsigned)((unsigned long long)(y < 0 ? -y : y) >> 24));
            }
          }
          rk *= rn;
          if (rk <= 0x1p-55f || term > 20) break;
          mx = __reduce_max_sync(0xffffffffu, mx);
          if (lane == 0) atomicMax(red + term, mx);
          mbar();  // also: every warp has read region B
          const int bits = 56 - __clz((int)red[term]);  // |E| < 2^bits
          sk = bits - kAccBits;
          lm = levels(sk);
          oz::put_planes<53, NE>(v, lm == 0 ? 1 : lm <= 2 ? 3 : 6, regB + own, PL, 6, half, bits - 53);
          mbar();
        }

        // 4. G' = the sum; Q <- -Q G'.
        const bool prod = !refl && n > a.inject_at;
        double2 q[NE];
        if (prod) {
          int eq0 = oz::kNoExp, eq1 = oz::kNoExp;
#pragma unroll
          for (int k = 0; k < NE; ++k) {
            q[k] = Qs[32 * k];
            if (erow(k)) eq1 = max(eq1, oz::fexp2(q[k]));
            else eq0 = max(eq0, oz::fexp2(q[k]));
          }
          oz::put_row_exps(exQ + (tj * NHALF + half) * MP, ti, lane, eq0, eq1);
        }
        mbar();  // region A and region B have been read
        // G' made exactly symmetric (below the diagonal from above it): left
        // to the rounding of the two halves, its asymmetry grew along the
        // guide and tripled the error of t.
        double2* gb = (double2*)regB;  // [MP][LDW]
        double2 gd[NE];
#pragma unroll
        for (int k = 0; k < NE; ++k) {
          const int e = (erow(k) ? ey1 : ey0) - kAccBits;
          const int i = r0 + erow(k), j = c0 + ecol(k);
          gd[k] = make_double2(oz::fix_to_double(acc[k], e), oz::fix_to_double(acc[NE + k], e));
          if (i < j) gb[i * LDW + j] = gd[k];
        }
        mbar();
#pragma unroll
        for (int k = 0; k < NE; ++k) {
          const int i = r0 + erow(k), j = c0 + ecol(k);
          if (i > j) gd[k] = gb[j * LDW + i];
          Gs[32 * k] = gd[k];
          if (prod) {
            acc[k] = oz::sfixed53(gd[k].x, erow(k) ? ey1 : ey0);
            acc[NE + k] = oz::sfixed53(gd[k].y, erow(k) ? ey1 : ey0);
          }
        }
        if (prod) {
          oz::put_planes<53, NE>(acc, 6, regA + own, PL, 6, half);
          mbar();  // region B has been read
        }
        if (prod) {
          const int eq0 = oz::row_exp<NCW>(exQ, MP, r0), eq1 = oz::row_exp<NCW>(exQ, MP, r0 + 8);
#pragma unroll
          for (int k = 0; k < NE; ++k) {
            const int e = erow(k) ? eq1 : eq0;
            acc[k] = oz::sfixed53(q[k].x, e);
            acc[NE + k] = oz::sfixed53(q[k].y, e);
          }
          oz::put_planes<53, NE>(acc, 6, regB + own, PL, 6, half);
          mbar();
#pragma unroll
          for (int h = 0; h < NE / 4; ++h) {
            long long hi[8], lo[8];
            oz::half_product<T, 6, 6, oz::kLmax>(bB + offA0, bB + offA1, 6 * kPlane, bA + offB + 8 * (odd ^ (half | h)),
                                                 6 * kPlane, kPlane, hi, lo);
#pragma unroll
            for (int w = 0; w < 4; ++w) {
              const int k = 4 * h + w;
              const int e = (erow(k) ? eq1 : eq0) + oz::row_exp<NCW>(exY, MP, c0 + ecol(k));
              Qs[32 * k] = make_double2(-oz::fold_to_double(hi[w], lo[w], e), -oz::fold_to_double(hi[4 + w], lo[4 + w], e));
            }
          }
        } else if (!refl) {
          // the source slice: Q = G'; zero before it
#pragma unroll
          for (int k = 0; k < NE; ++k) Qs[32 * k] = n == a.inject_at ? Gs[32 * k] : make_double2(0.0, 0.0);
        }
        if (a.state_dump) {
          // The state after this slice, natural order: Gss = w G' w and
          // Gs1 = w Q^T w, the solve_block_tridiag pair (S_n, Z_n).
          double2* d1 = a.state_dump + ((int64_t)r * nx + n) * 2 * M * M;
#pragma unroll
          for (int k = 0; k < NE; ++k) {
            const int i = r0 + erow(k), j = c0 + ecol(k);
            if (i < M && j < M) {
              d1[(int64_t)i * M + j] = cmul(Ww[32 * k], Gs[32 * k]);
              d1[(int64_t)M * M + (int64_t)j * M + i] = cmul(Ww[32 * k], Qs[32 * k]);
            }
          }
        }
      }
    }
    __syncthreads();

    if (s_status == kStatusNeedPivot) {
      if (tid == 0) {
        a.status[r] = kStatusNeedPivot;
        a.flag_list[atomicAdd(a.work_counter + 1, 1)] = r;
      }
      __syncthreads();
      continue;
    }

    if (refl) {
      // Reflection from the reverse sweep: r = -1 + 2i sqrt(real mu) G11
      // sqrt(real mu) (src/waveguide.f90:510-512), G11 = w G' w.
      double2* rout = a.tout + (int64_t)r * M * M;
      if (main_thread) {
#pragma unroll
        for (int k = 0; k < NE; ++k) {
          const int i = r0 + erow(k), j = c0 + ecol(k);
          if (i < M && j < M) {
            const double2 v = cmul(cmul(wd.sqmu_r[i], cmul(Ww[32 * k], Gs[32 * k])), wd.sqmu_r[j]);
            rout[i + (int64_t)j * M] = make_double2((i == j ? -1.0 : 0.0) - 2.0 * v.y, 2.0 * v.x);
          }
        }
      }
      __syncthreads();
      if (tid == 0) a.status[r] = s_status;
      continue;
    }

    // 5. Fisher-Lee, t = 2i sqmu Gs1 sqmu with Gs1 = w Q^T w, into region A
    //    (free now) for the eigenvalue stage.
    double2* W = (double2*)regA;  // [MP][LDW]
    const int row0 = tmat ? 0 : wd.row0, col0 = tmat ? 0 : wd.col0;
    const int nrow = tmat ? M : wd.nrow, ncol = tmat ? M : wd.ncol;
    const double2* sqmu = tmat ? wd.sqmu_r : wd.sqmu_c;
    double2* tout = a.tout ? a.tout + (int64_t)r * nrow * ncol : nullptr;
    if (main_thread) {
#pragma unroll
      for (int k = 0; k < NE; ++k) {
        const int gj = r0 + erow(k), gi = c0 + ecol(k);  // Q[j][i]
        const int i = gi - row0, j = gj - col0;
        if (i >= 0 && i < nrow && j >= 0 && j < ncol) {
          const double2 v = cmul(cmul(sqmu[gi], cmul(Ww[32 * k], Qs[32 * k])), sqmu[gj]);
          const double2 tv = make_double2(-2.0 * v.y, 2.0 * v.x);
          if (tout) tout[i + (int64_t)j * nrow] = tv;
          W[i * LDW + j] = tv;
        }
      }
    }
    __syncthreads();
    if (!tmat) {
      // 6. Eigenvalues of t^H t, sorted descending into teig.
      const int64_t obase = a.teig_off ? a.teig_off[r] : (int64_t)r * wd.neigv;
      tt_eigenvalues<NT>(W, LDW, nrow, ncol, wd.neigv, cc, a.teig + obase);
    }
    __syncthreads();
    if (tid == 0) a.status[r] = s_status;
  }
}

template <int T>
int plan_sym_t(SweepArgs& a, int sm_count, int* grid, int64_t* stride) {
  const size_t smem = SymCfg<T>::bytes();
  RG_CUDA(allow_smem((const void*)sweep_sym_kernel<T>, smem));
  int per_sm = 0;
  RG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sweep_sym_kernel<T>, SymCfg<T>::NT, smem));
  if (per_sm < 1) return fail(RG_ERR_INVALID_ARG, "symmetric sweep kernel does not fit on an SM");
  if (a.force_per_sm > 0 && a.force_per_sm < per_sm) per_sm = a.force_per_sm;
  int g = per_sm * sm_count;
  if (g > a.nreal) g = a.nreal;
  *grid = g < 1 ? 1 : g;
  *stride = sym_stride(T, a.max_ny);
  a.cluster = 1;
  return RG_OK;
}

template <int T>
int launch_sym_t(const SweepArgs& a, cudaStream_t stream, int grid) {
  sweep_sym_kernel<T><<<grid, SymCfg<T>::NT, SymCfg<T>::bytes(), stream>>>(a);
  RG_CUDA(cudaGetLastError());
  return RG_OK;
}

}  // namespace

int sweep_sym_plan(SweepArgs& a, int sm_count, int* grid, int64_t* work_stride) {
  if (a.max_M <= 16) return plan_sym_t<1>(a, sm_count, grid, work_stride);
  if (a.max_M <= 32) return plan_sym_t<2>(a, sm_count, grid, work_stride);
  if (a.max_M <= 48) return plan_sym_t<3>(a, sm_count, grid, work_stride);
  if (a.max_M <= kMaxModesSmem) return plan_sym_t<4>(a, sm_count, grid, work_stride);
  return fail(RG_ERR_INVALID_ARG, "symmetric sweep kernel: too many modes");
}

int launch_sweep_sym(const SweepArgs& a, cudaStream_t stream, int grid) {
  if (a.nreal <= 0) return RG_OK;
  if (a.max_M <= 16) return launch_sym_t<1>(a, stream, grid);
  if (a.max_M <= 32) return launch_sym_t<2>(a, stream, grid);
  if (a.max_M <= 48) return launch_sym_t<3>(a, stream, grid);
  return launch_sym_t<4>(a, stream, grid);
}

}  // namespace rg
