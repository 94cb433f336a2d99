// The inverse of a complex symmetric matrix of up to 16 T modes by one CTA,
// to FP64 accuracy without FP64 elimination: the core of the sweep of up to 64
// modes (rg_sweep_sym.cu), and the leaf blocks of the sweep above
// (rg_sweep_large_sym.cu).
//
//   1. Y0 = X^-1 in FP32 (block Gauss-Jordan on the 16 x 16 tiles that the
//      warps hold in registers), rounded to 26-bit fixed point;
//   2. its residual R = I - Y0 X exactly enough (2^-58), on the FP16 tensor
//      cores with the balanced 9-bit digits of rg_ozaki.cuh, seven of them
//      for X (with six, its rounding relative to the row's largest entry
//      doubled the error of t);
//   3. G = (I + R + R^2 + ...) Y0: E_1 = R Y0, E_k+1 = R E_k, summed in
//      64-bit fixed point until ||R||^(k+1) is below 2^-55.  ||R|| is near
//      1e-5, so three terms do, and the digits kept in each follow from the
//      magnitudes.
//
// FP64 is 1.7 FMA lanes per clock and SM here; no FP64 instruction is left.
// 58,000 clocks at 32 modes, 180,000 at 64 (an FP64 elimination: 150,000 and
// 300,000 at 32 and 64 modes by 8 warps).  Bound by its serial chains: the
// pivots of the FP32 part, two thirds of the time at 32 modes, and the mma and
// barriers of the products.
//
// Layout: T tiles a side, a warp per tile (ti, tj), or two warps with a column
// half each, in the accumulator layout of mma.m16n8k16, which for two n8 tiles
// is also the fragment layout of its A operand and, read as the transpose, of
// its B operand: digits go from registers to shared memory and back without a
// shuffle, and one set of planes serves both sides of a symmetric matrix.  Two
// plane regions of 12 x T^2 x 512 bytes are reused:
//   region A: X -> R;   region B: Y0 -> E_k.
#pragma once

#include "rg_device.cuh"
#include "rg_ozaki.cuh"

namespace rg {

// Fixed point: Y0 has 26 bits, the sum of the series 56, relative to the
// power of two of the row.
constexpr int kY0Bits = 26, kAccBits = 56;

// Pivots of the FP32 elimination come in natural order, and the residual of
// its result is checked, so they may be this much smaller against their row
// than sym_tau asks of a pivot that was searched for.
constexpr double kNaturalTau = 0.1;

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

__device__ __forceinline__ void fms(float2& m, float2 f, float2 s) {  // m -= f s
  m.x = fmaf(f.y, s.y, fmaf(-f.x, s.x, m.x));
  m.y = fmaf(-f.y, s.x, fmaf(-f.x, s.y, m.y));
}

// Entry k of a lane: row g + erow(k), column 2 t + ecol(k) (plus 8 in the
// second half of a split tile), with g = lane / 4, t = lane % 4.
__device__ __forceinline__ constexpr int erow(int k) { return 8 * ((k >> 1) & 1); }
__device__ __forceinline__ constexpr int ecol(int k) { return (k & 1) + 8 * (k >> 2); }

// A published FP32 tile: rows of 18 complex, so that the eight rows a warp
// reads at once lie in different banks.
constexpr int kTileLd = 18, kTileF2 = 16 * kTileLd;

// m -= A B over the 16 columns of A, for a lane's entries (rows g, g + 8;
// columns lc, lc + 1 and, for a whole tile, 8 further on).  (Packed FMAs, two to
// an instruction, need as many moves for their swapped and negated pairs.)
template <int NE>
__device__ __forceinline__ void tile_fms(float2* m, const float2* A, const float2* B, int g, int lc) {
#pragma unroll 2
  for (int k = 0; k < 16; ++k) {
    const float2 f0 = A[g * kTileLd + k], f1 = A[(g + 8) * kTileLd + k];
#pragma unroll
    for (int q = 0; q < NE; q += 4) {
      const float4 u = *reinterpret_cast<const float4*>(B + k * kTileLd + lc + 2 * q);
      fms(m[q], f0, make_float2(u.x, u.y));
      fms(m[q + 1], f0, make_float2(u.z, u.w));
      fms(m[q + 2], f1, make_float2(u.x, u.y));
      fms(m[q + 3], f1, make_float2(u.z, u.w));
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

template <int N>
struct Int {
  static constexpr int value = N;
};

// The shared memory of tile_inverse: the plane regions (12 planes of T^2 x 32
// uint4 each), [32] maxima, one sum, and two [NCW][16 T] arrays of row
// exponents by warp column (of X and of Y0; the latter also scale the
// result's fixed point in the caller).
struct TileSmem {
  uint4* regA;
  uint4* regB;
  unsigned* red;
  unsigned long long* rsum;
  int* exX;
  int* exY;
};

// x: this lane's entries of X (zero outside M x M), NE = 8 of a whole tile or
// 4 of its column half, real parts, then imaginary parts; gd: its entries of
// X^-1, exactly symmetric; ey0, ey1: the exponents of rows g and g + 8 (|gd| <=
// 2^ey (1 + 2^-9)).  With NP = 2 (T = 1) a lane has one part of its entries, real
// in even warps and imaginary in odd ones: half the instructions in each of twice
// the warps.  Called by the T^2 8/NE NP warps 0, 1, ... of the CTA; bar() is a
// barrier of theirs, and pre() is run before the last but one.  Returns false, in
// every thread, when a pivot falls below tau times the largest unswept entry of
// its row (in its tile) or the residual is not small; *flag (shared, zero before,
// kStatusNeedPivot after) says so too.  *late becomes kStatusNeedPivot before the
// last barrier when the result is useless because an entry of a term or of the
// inverse does not fit the fixed point that Y0 gave its row (the caller looks at
// it after the last slice: a read here would lengthen every slice by a barrier's
// latency).  Unchecked, that gave T up to 7000 in one of some 1000 realizations
// of 20 to 64 modes under strong disorder.
template <int T, int NE, int NP = 1, class Bar, class Pre>
__device__ __forceinline__ bool tile_inverse(const double* x, const int M, const float tau, const TileSmem& s,
                                             volatile int* flag, volatile int* late, Bar bar, Pre pre, double* gd,
                                             int& ey0, int& ey1) {
  static_assert(NP == 1 || T == 1, "a part each only for one tile");
  constexpr int MP = 16 * T, NV = 2 * NE / NP, NHALF = 8 / NE, NCW = T * NHALF * NP, PL = T * T * 32, LDW = MP + 1;
  const int tid = threadIdx.x, lane = tid & 31, warp = (tid >> 5) / NP, part = NP == 2 ? (tid >> 5) & 1 : 0;
  const int cw = (warp % (T * NHALF)) * NP + part;  // this warp among those of its rows
  const int g = lane >> 2, t4 = lane & 3;
  const int tile = warp / NHALF, half = NHALF == 2 ? warp & 1 : 0;
  const int ti = tile / T, tj = tile % T;
  const int r0 = ti * 16 + g, c0 = tj * 16 + 2 * t4 + 8 * half;
  uint4 *const regA = s.regA, *const regB = s.regB;
  unsigned* const red = s.red;
  unsigned long long* const rsum = s.rsum;
  int *const exX = s.exX, *const exY = s.exY;
  // This lane's place in the planes: its tile, and the word pairs of its tile
  // row (as A) and tile column (as B), in bytes.
  constexpr int kPlane = 16 * PL;
  const int odd = (lane >> 3) & 1;
  const int own = tile * 32 + lane;
  const int offA0 = ti * T * 512 + lane * 16 + 8 * odd, offA1 = ti * T * 512 + lane * 16 + 8 * (1 - odd);
  const int offB = tj * T * 512 + lane * 16;
  const char* bA = (const char*)regA;
  const char* bB = (const char*)regB;

  // Row exponents over the warps of a row, then the planes of X.
  float2 m[NE];  // (NP = 2: the other part is not used)
  uint32_t x7[NE / NP];  // the seventh digit of X
  {
    int e0 = oz::kNoExp, e1 = oz::kNoExp;
#pragma unroll
    for (int k = 0; k < NE; ++k) {
      const int e = oz::fexp2(make_double2(x[k], NP == 1 ? x[NE + k] : 0.0));
      if (erow(k)) e1 = max(e1, e);
      else e0 = max(e0, e);
    }
    oz::put_row_exps(exX + cw * MP, ti, lane, e0, e1);
    bar();
    if (tid < 32) red[tid] = 0;
    if (tid == 0) rsum[0] = 0;
    e0 = oz::row_exp<NCW>(exX, MP, r0);
    e1 = oz::row_exp<NCW>(exX, MP, r0 + 8);
    long long fx[NV];
#pragma unroll
    for (int k = 0; k < NE; ++k) {
      const int e = erow(k) ? e1 : e0;
      fx[k] = oz::sfixed62(x[k], e);
      m[k].x = to_f32(x[k]);
      if (NP == 1) {
        fx[NV - NE + k] = oz::sfixed62(x[NV - NE + k], e);
        m[k].y = to_f32(x[NV - NE + k]);
      }
    }
    oz::put_planes<62, NE, NP>(fx, 6, regA + own, PL, 6, half, 0, x7, part);
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
    for (int q = 0; q < NE; q += 2) {
      float2* d = dst + (g + erow(q)) * kTileLd + lc + (q & 4 ? 8 : 0);
      if (NP == 2) {
        reinterpret_cast<float*>(d)[part] = m[q].x;
        reinterpret_cast<float*>(d)[2 + part] = m[q + 1].x;
      } else {
        *reinterpret_cast<float4*>(d) = make_float4(m[q].x, m[q].y, m[q + 1].x, m[q + 1].y);
      }
    }
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
    bar();
    if (ti == t && tj == t && half == 0 && part == 0) small_pivot |= invert_tile(Pt, min(16, M - 16 * t), tau, lane);
    bar();
    if (ti == t && tj == t) {
#pragma unroll
      for (int q = 0; q < NE; ++q) {
        m[q] = Pt[(g + erow(q)) * kTileLd + lc + ecol(q)];
        if (NP == 2 && part) m[q].x = m[q].y;
      }
    } else if (T > 1 && (ti == t || tj == t)) {
#pragma unroll
      for (int q = 0; q < NE; ++q) m[q] = make_float2(0.0f, 0.0f);
      tile_fms<NE>(m, ti == t ? Pt : Ct + ti * kTileF2, ti == t ? Rt + tj * kTileF2 : Pt, g, lc);
      if (ti == t) {
#pragma unroll
        for (int q = 0; q < NE; ++q) m[q] = make_float2(-m[q].x, -m[q].y);
        put_tile(St + tj * kTileF2);
      }
    }
    if (T > 1) {
      bar();
      if (ti != t && tj != t) tile_fms<NE>(m, Ct + ti * kTileF2, St + tj * kTileF2, g, lc);
      bar();
    }
  }
  if (small_pivot) *flag = kStatusNeedPivot;
  // Y0 made exactly symmetric (the entries below the diagonal from
  // above it), so that its planes serve as both operands.
  float2* sy = (float2*)(regB + 6 * PL);  // [MP][LDW]
#pragma unroll
  for (int k = 0; k < NE; ++k) {
    float2* d = sy + (r0 + erow(k)) * LDW + c0 + ecol(k);
    if (NP == 2) reinterpret_cast<float*>(d)[part] = m[k].x;
    else *d = m[k];
  }
  bar();
  if (*flag == kStatusNeedPivot) return false;
#pragma unroll
  for (int k = 0; k < NE; ++k) {
    const int i = r0 + erow(k), j = c0 + ecol(k);
    if (i > j) {
      m[k] = sy[j * LDW + i];
      if (NP == 2 && part) m[k].x = m[k].y;
    }
    if (NP == 2) m[k].y = 0.0f;
  }
  long long acc[NV];  // the sum of the series, kAccBits of the row's power of two
  {
    unsigned k0 = 0, k1 = 0;
#pragma unroll
    for (int k = 0; k < NE; ++k) {
      if (erow(k)) k1 = max(k1, fkey(m[k]));
      else k0 = max(k0, fkey(m[k]));
    }
    oz::put_row_exps(exY + cw * MP, ti, lane, k0 ? (int)(k0 >> 23) - 126 : oz::kNoExp,
                     k1 ? (int)(k1 >> 23) - 126 : oz::kNoExp);
    bar();
    ey0 = oz::row_exp<NCW>(exY, MP, r0);
    ey1 = oz::row_exp<NCW>(exY, MP, r0 + 8);
    // 2^(26 - e) as a float (e within +-100; anything else is flagged by the residual)
    const float s0 = __uint_as_float((unsigned)(127 + kY0Bits - max(-100, min(100, ey0))) << 23);
    const float s1 = __uint_as_float((unsigned)(127 + kY0Bits - max(-100, min(100, ey1))) << 23);
#pragma unroll
    for (int k = 0; k < NE; ++k) {
      const float f = erow(k) ? s1 : s0;
      acc[k] = __float2int_rn(m[k].x * f);
      if (NP == 1) acc[NV - NE + k] = __float2int_rn(m[k].y * f);
    }
    oz::put_planes<kY0Bits, NE, NP>(acc, 3, regB + own, PL, 3, half, 0, nullptr, part);
    oz::put_words<NE>(x7, regB + (6 + part) * PL + own, odd, half);
    if (NP == 1) oz::put_words<NE>(x7 + (NE / 2) % (NE / NP), regB + 7 * PL + own, odd, half);
#pragma unroll
    for (int k = 0; k < NV; ++k) acc[k] *= 1LL << (kAccBits - kY0Bits);
  }
  bar();

  // 3. R = I - Y0 X at 2^-62, its largest entry and Frobenius norm.
  long long v[NV];
  unsigned mx = 0;
  unsigned long long sq = 0;
#pragma unroll
  for (int h = 0; h < NE / 4; ++h) {
    long long hi[8], lo[8];
    oz::half_product<T, 3, 7, oz::kLmax, NP>(bB + offA0, bB + offA1, 3 * kPlane, bA + offB + 8 * (odd ^ (half | h)),
                                         6 * kPlane, kPlane, hi, lo,
                                         bB + 6 * kPlane + offB + 8 * (odd ^ (half | h)), part);
#pragma unroll
    for (int w = 0; w < 8 / NP; ++w) {
      const int k = 4 * h + (w & 3);
      const int i = r0 + erow(k), j = c0 + ecol(k);
      const int e = (erow(k) ? ey1 : ey0) + oz::row_exp<NCW>(exX, MP, j);
      long long y = 0;
      if (i < M && j < M) {
        const int up = 35 - e;  // |Y0 X| < 2, or the inverse is useless
        const long long top = hi[w] + (lo[w] >> 36);
        const bool fits = up >= 62 || (up >= 0 ? (top >> up) == 0 || (top >> up) == -1 : top == 0);
        y = (w < 4 && part == 0 && i == j ? 1LL << 62 : 0) - oz::fix_shift(hi[w], lo[w], 28 + e);
        const unsigned long long av = (unsigned long long)(y < 0 ? -y : y);
        mx = max(mx, fits ? (unsigned)(av >> 32) : ~0u);
        const unsigned long long q = min(av >> 36, 1ULL << 26);
        sq += q * q;
      }
      v[(w < 4 ? 0 : NE) + k] = i < M && j < M ? 2 * y - 1 : 0;  // (fix_shift truncates: half a unit taken back)
    }
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
#pragma unroll
  for (int off = 16; off; off >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, off);
  if (lane == 0) {
    atomicMax(red, mx);
    atomicAdd(rsum, sq);
  }
  bar();
  const int er = 2 - __clz((int)red[0]);  // |R| < 2^er (at least 2^-30)
  const float rn = sqrtf((float)rsum[0]) * 0x1p-26f + (float)M * 0x1p-25f;
  if (!(rn < 0.125f) || er > -2) {
    if (tid == 0) *flag = kStatusNeedPivot;
    return false;
  }
  // Levels of a product of R with a matrix below 2^s of its row's power
  // of two: the dropped ones stay below 2^-57 of it.
  auto levels = [&](int s) { return max(0, min(oz::kLmax, (62 + er + s + 8) / 9 - 1)); };
  // E_1 = R Y0, E_k+1 = R E_k; the sum starts from Y0.
  int lm = levels(0);
  oz::put_planes<53, NE, NP>(v, 6, regA + own, PL, 6, half, 10 + er, nullptr, part);
  bar();
  bool bad = false;  // an entry does not fit its row's fixed point
  // rows' exponents, those of the padding (where all is zero) out of the way
  const int eu0 = r0 < M ? ey0 : 1 << 14, eu1 = r0 + 8 < M ? ey1 : 1 << 14;
  float rk = rn;  // ||R||^k of the term just formed
  int sk = 0;     // the B operand's entries are below 2^(e_i + sk)
  for (int term = 1;; ++term) {
    mx = 0;
#pragma unroll
    for (int h = 0; h < NE / 4; ++h) {
      long long hi[8], lo[8];
      const char* b = bB + offB + 8 * (odd ^ (half | h));
      // the digits that the levels 0 .. lm take
      if (term == 1) {
        if (lm <= 4)
          oz::half_product<T, 5, 3, 4, NP>(bA + offA0, bA + offA1, 6 * kPlane, b, 3 * kPlane, kPlane, hi, lo, nullptr,
                                           part);
        else if (lm == 5)
          oz::half_product<T, 6, 3, 5, NP>(bA + offA0, bA + offA1, 6 * kPlane, b, 3 * kPlane, kPlane, hi, lo, nullptr,
                                           part);
        else
          oz::half_product<T, 6, 3, 6, NP>(bA + offA0, bA + offA1, 6 * kPlane, b, 3 * kPlane, kPlane, hi, lo, nullptr,
                                           part);
      } else {
        auto product = [&](auto n, auto lmax) {
          oz::half_product<T, decltype(n)::value, decltype(n)::value, decltype(lmax)::value, NP>(
              bA + offA0, bA + offA1, 6 * kPlane, b, 6 * kPlane, kPlane, hi, lo, nullptr, part);
        };
        if (lm == 0) product(Int<1>{}, Int<0>{});
        else if (lm == 1) product(Int<2>{}, Int<1>{});
        else if (lm == 2) product(Int<3>{}, Int<2>{});
        else if (lm <= 4) product(Int<5>{}, Int<4>{});
        else product(Int<6>{}, Int<6>{});
      }
      int e[4], top = oz::kNoExp;
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        e[w] = er + sk + oz::row_exp<NCW>(exY, MP, c0 + ecol(4 * h + w)) - (erow(w) ? eu1 : eu0);
        top = max(top, e[w]);
      }
      // However small ||R|| is, R Y0 brings entries of a large row of Y0 to a
      // small one: |E| must stay below 2^4 of the row's power of two.  It does
      // where e < -8, as |hi| < 2^46; else every entry is looked at (for one tile
      // always: there the latency of a branch costs more than its instructions).
      if (T == 1 || top >= -8) {
#pragma unroll
        for (int w = 0; w < 8 / NP; ++w)
          bad |= (unsigned long long)(((hi[w] + (lo[w] >> 36)) >> min(max(94 - kAccBits - e[w & 3], 0), 63)) + 1) > 1;
      }
#pragma unroll
      for (int w = 0; w < 8 / NP; ++w) {
        // rounded: truncating, a bias of 2^-57 in every entry, is an
        // error of M 2^-57 in norm that adds up from slice to slice
        const long long y = (oz::fix_shift(hi[w], lo[w], kAccBits - 33 + e[w & 3]) + 1) >> 1;
        const int q = (w < 4 ? 0 : NE) + 4 * h + (w & 3);
        acc[q] += y;
        v[q] = y;
        mx = max(mx, (unsigned)((unsigned long long)(y < 0 ? -y : y) >> 24));
      }
    }
    rk *= rn;
    if (rk <= 0x1p-55f || term > 20) break;
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) atomicMax(red + term, mx);
    bar();  // also: every warp has read region B
    const int bits = 56 - __clz((int)red[term]);  // |E| < 2^bits
    sk = bits - kAccBits;
    lm = levels(sk);
    oz::put_planes<53, NE, NP>(v, lm <= 2 ? lm + 1 : lm <= 4 ? 5 : 6, regB + own, PL, 6, half,
                                  bits - 53, nullptr, part);
    bar();
  }

  pre();
  bar();  // region A and region B have been read
  // G made exactly symmetric (below the diagonal from above it): left
  // to the rounding of the two halves, its asymmetry grew along the
  // guide and tripled the error of t.
  double* gb = (double*)regB;  // [MP][LDW] complex
  constexpr int kTop = (1 << (kAccBits - 32)) + (1 << (kAccBits - 41));
  unsigned most = 0;
#pragma unroll
  for (int k = 0; k < NE; ++k) {
    const int e = (erow(k) ? ey1 : ey0) - kAccBits;
    const int i = r0 + erow(k), j = c0 + ecol(k);
#pragma unroll
    for (int q = k; q < NV; q += NE) {
      gd[q] = oz::fix_to_double(acc[q], e);
      // the callers' digits hold entries of a row up to 2^ey (1 + 2^-8)
      most = max(most, (unsigned)((int)(acc[q] >> 32) + kTop));
      if (i < j) gb[2 * (i * LDW + j) + (q < NE ? part : 1)] = gd[q];
    }
  }
  if (bad || most > 2u * kTop) *late = kStatusNeedPivot;
  bar();
#pragma unroll
  for (int k = 0; k < NE; ++k) {
    const int i = r0 + erow(k), j = c0 + ecol(k);
#pragma unroll
    for (int q = k; q < NV; q += NE)
      if (i > j) gd[q] = gb[2 * (j * LDW + i) + (q < NE ? part : 1)];
  }
  return true;
}

}  // namespace rg
