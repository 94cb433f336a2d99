// Complex FP64 matrix products on the FP16 tensor cores in modular arithmetic.
//
// C = A B for M x M complex matrices (M <= 512), mma.sync m16n8k16 (FP16
// inputs, FP32 accumulation), with the accuracy of an exact product of the
// operands rounded to 53-bit fixed point:
//
//  * row i of A has the exponent ea_i of its largest |re| or |im| (|A_ik| <
//    2^ea_i), column j of B the exponent eb_j; entries are rounded to the
//    integers X = A_ik 2^(53-ea_i), |X| <= 2^53 (as in rg_ozaki.cuh);
//  * the integer product |C'| <= 2 M 2^106 <= 2^116 is recovered from its
//    residues modulo 12 coprime moduli p <= 1021 whose product P exceeds
//    2^119 (Chinese remainder theorem);
//  * every prime factor of every p is 1 mod 4, so -1 has a square root s
//    modulo p, and (a + i b) -> (u, v) = (a + s b, a - s b) turns the complex
//    product modulo p into two real ones: u_C = u_A u_B, v_C = v_A v_B.  24
//    real products of M^3 in all, where 26 digit pairs with four real products
//    each take 104;
//  * residues are balanced, |r| <= 511, exact in FP16; sums over 64 k stay
//    below 64 511^2 + 511 < 2^24, so they are exact in FP32, and are reduced
//    modulo p after every 64 k;
//  * a_m = (C' (P/p_m)^-1) mod p_m for both parts comes from u and v by one
//    constant each, and C' = sum_m a_m P/p_m - k P with k = the nearest
//    integer to sum_m a_m / p_m (|C'| < P/8, so an FP32 sum decides it).  The
//    sum is formed in 96-bit integers in units of 2^23 (error below 2^36, 2^-70
//    of 2^106), then rounded to FP64 once.
//
// The result depends on neither tiling nor order.  What it replaces in the
// blocked sweep is the digit loop (oz::gemm_block): 7.5k clocks per 32 x 64
// block and 16 k with two CTAs on an SM, bound by instructions around the mma
// (1,400 a warp for 208), the folds of the level sums above all.
//
// Layouts: fragment order as in rg_ozaki.cuh.  An operand's planes: uint4 [12
// moduli][u, v][T row (A) or column (B) tiles][T k tiles][32 lanes].
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>

#include "rg_ozaki.cuh"

namespace rg {
namespace crt {

constexpr int kMod = 12;
constexpr int kUnit = 23;  // C' is summed in units of 2^kUnit

__host__ __device__ inline int64_t operand_uint4(int M) {
  const int64_t T = oz::tiles(M);
  return 2LL * kMod * T * T * 32;
}
// Scratch of one CTA for the residues of a 64 x 64 block, in uint4.
constexpr int64_t kBlockUint4 = 2LL * kMod * 16 * 32;

struct Tables {
  float p[kMod], inv[kMod];     // modulus and its reciprocal
  float c[kMod][3];             // 2^14, 2^28, 2^42 mod p
  float s[kMod][4];             // s 2^(14 j) mod p
  float k1[kMod], k2[kMod];     // a_re = (u + v) k1, a_im = (u - v) k2 mod p
  uint32_t g[kMod][3];          // P / p / 2^kUnit, rounded, 32-bit words from the lowest
  uint32_t q[3];                // P / 2^kUnit, rounded
  uint32_t off[3];              // sum over m of 1024 g, modulo 2^96
};

typedef unsigned __int128 u128;

constexpr int kModuli[kMod] = {1021, 1013, 1009, 997, 985, 977, 953, 949, 941, 937, 929, 901};

constexpr int balanced(long long x, int p) {
  int r = (int)(x % p);
  if (r < 0) r += p;
  return r > p / 2 ? r - p : r;
}
constexpr int inverse(int a, int p) {
  a = ((a % p) + p) % p;
  for (int x = 1; x < p; ++x)
    if ((long long)a * x % p == 1) return x;
  return 0;
}
constexpr int root_of_minus_one(int p) {
  for (int x = 1; x < p; ++x)
    if ((long long)x * x % p == p - 1) return x;
  return 0;
}

constexpr Tables make_tables() {
  Tables t{};
  u128 P = 1;
  for (int m = 0; m < kMod; ++m) P *= (u128)kModuli[m];
  u128 off = 0;
  for (int m = 0; m < kMod; ++m) {
    const int p = kModuli[m];
    const u128 Pm = P / (u128)p;
    const int inv = inverse((int)(Pm % (u128)p), p), s = root_of_minus_one(p);
    t.p[m] = (float)p;
    t.inv[m] = 1.0f / (float)p;
    for (int j = 0; j < 4; ++j) {
      const int c = balanced(1LL << (14 * j), p);
      if (j > 0) t.c[m][j - 1] = (float)c;
      t.s[m][j] = (float)balanced((long long)c * s, p);
    }
    t.k1[m] = (float)balanced((long long)inv * inverse(2, p), p);
    t.k2[m] = (float)balanced((long long)inv * inverse(2 * s, p), p);
    const u128 gm = (Pm + ((u128)1 << (kUnit - 1))) >> kUnit;
    for (int w = 0; w < 3; ++w) t.g[m][w] = (uint32_t)(gm >> (32 * w));
    off += gm * 1024;
  }
  const u128 q = (P + ((u128)1 << (kUnit - 1))) >> kUnit;
  for (int w = 0; w < 3; ++w) {
    t.q[w] = (uint32_t)(q >> (32 * w));
    t.off[w] = (uint32_t)(off >> (32 * w));
  }
  return t;
}
static __constant__ Tables kT = make_tables();

constexpr float kMagic = 12582912.0f;  // 1.5 2^23: x + kMagic rounds x to an integer in the low bits

// Two FP32 operations in one instruction, on the pair of a word's entries.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  unsigned long long x, y, z, r;
  memcpy(&x, &a, 8);
  memcpy(&y, &b, 8);
  memcpy(&z, &c, 8);
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(x), "l"(y), "l"(z));
  float2 o;
  memcpy(&o, &r, 8);
  return o;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  unsigned long long x, y, r;
  memcpy(&x, &a, 8);
  memcpy(&y, &b, 8);
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
  float2 o;
  memcpy(&o, &r, 8);
  return o;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  unsigned long long x, y, r;
  memcpy(&x, &a, 8);
  memcpy(&y, &b, 8);
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
  float2 o;
  memcpy(&o, &r, 8);
  return o;
}
__device__ __forceinline__ float2 both(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 reduce2(float2 x, float2 mp, float2 inv) {  // mp = -p
  const float2 q = add2(fma2(x, inv, both(kMagic)), both(-kMagic));
  return fma2(q, mp, x);
}

__device__ __forceinline__ float reduce(float x, float p, float inv) {
  const float q = fmaf(x, inv, kMagic) - kMagic;
  return fmaf(-q, p, x);
}

// Balanced base-2^14 limbs of a signed integer below 2^53 + 1, as floats.
__device__ __forceinline__ void limbs(long long x, float f[4]) {
  const long long bias = 8192LL * (1 + (1LL << 14) + (1LL << 28));
  const unsigned long long y = (unsigned long long)(x + bias + (8192LL << 42));
#pragma unroll
  for (int j = 0; j < 3; ++j)
    f[j] = __uint_as_float(0x4B000000u | ((uint32_t)(y >> (14 * j)) & 16383u)) - (8388608.0f + 8192.0f);
  f[3] = __uint_as_float(0x4B000000u | (uint32_t)(y >> 42)) - (8388608.0f + 8192.0f);
}

__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  uint32_t r;
  memcpy(&r, &h, 4);
  return r;
}

// x 2^(53-e) rounded to nearest, with sign (|x| < 2^e).
__device__ __forceinline__ long long fixed(double x, int e) {
  const long long m = (long long)oz::fixed53(x, e);
  return x < 0.0 ? -m : m;
}

// The 24 planes' uint4 of one lane of one tile from its 8 complex entries in
// fragment order and their exponents; dst points at [modulus 0][u][this
// tile][lane], `plane` uint4 between planes.
__device__ __forceinline__ void write_residues(const double2 v[8], const int e[8], uint4* dst, int64_t plane) {
  float2 xr[4][4], xi[4][4];  // [word][limb]
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    float r0[4], r1[4], i0[4], i1[4];
    limbs(fixed(v[2 * k].x, e[2 * k]), r0);
    limbs(fixed(v[2 * k + 1].x, e[2 * k + 1]), r1);
    limbs(fixed(v[2 * k].y, e[2 * k]), i0);
    limbs(fixed(v[2 * k + 1].y, e[2 * k + 1]), i1);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      xr[k][j] = make_float2(r0[j], r1[j]);
      xi[k][j] = make_float2(i0[j], i1[j]);
    }
  }
#pragma unroll 1
  for (int m = 0; m < kMod; ++m) {
    const float2 mp = both(-kT.p[m]), inv = both(kT.inv[m]);
    const float2 c1 = both(kT.c[m][0]), c2 = both(kT.c[m][1]), c3 = both(kT.c[m][2]);
    const float2 s0 = both(kT.s[m][0]), s1 = both(kT.s[m][1]), s2 = both(kT.s[m][2]), s3 = both(kT.s[m][3]);
    uint32_t u[4], w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 x = fma2(xr[k][3], c3, fma2(xr[k][2], c2, fma2(xr[k][1], c1, xr[k][0])));
      const float2 y = reduce2(fma2(xi[k][3], s3, fma2(xi[k][2], s2, fma2(xi[k][1], s1, mul2(xi[k][0], s0)))), mp, inv);
      const float2 a = reduce2(add2(x, y), mp, inv), b = reduce2(fma2(y, both(-1.0f), x), mp, inv);
      u[k] = pack_half2(a.x, a.y);
      w[k] = pack_half2(b.x, b.y);
    }
    __stcg(dst + (2 * m) * plane, make_uint4(u[0], u[1], u[2], u[3]));
    __stcg(dst + (2 * m + 1) * plane, make_uint4(w[0], w[1], w[2], w[3]));
  }
}

// Residue planes of A: entries A(i, k) = getA(i, k) (zero outside M x M),
// exponents ea[i].  Task = (row tile, k tile, lane), from task0 by `step`.
template <class GetA>
__device__ void split_a(int M, GetA getA, const int* ea, uint4* dig, int task0, int step) {
  const int T = oz::tiles(M);
  const int64_t plane = (int64_t)T * T * 32;
  for (int task = task0; task < T * T * 32; task += step) {
    const int lane = task & 31, tk = (task >> 5) % T, ti = (task >> 5) / T;
    const int r0 = ti * 16 + (lane >> 2), k0 = tk * 16 + 2 * (lane & 3);
    double2 v[8];
    int e[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int r = r0 + 8 * ((k >> 1) & 1), c = k0 + (k & 1) + 8 * (k >> 2);
      v[k] = r < M && c < M ? getA(r, c) : make_double2(0.0, 0.0);
      e[k] = r < M ? ea[r] : 0;
    }
    write_residues(v, e, dig + ((int64_t)ti * T + tk) * 32 + lane, plane);
  }
}

// Residue planes of B: entries B(k, j) = getB(k, j), exponents eb[j].
template <class GetB>
__device__ void split_b(int M, GetB getB, const int* eb, uint4* dig, int task0, int step) {
  const int T = oz::tiles(M);
  const int64_t plane = (int64_t)T * T * 32;
  for (int task = task0; task < T * T * 32; task += step) {
    const int lane = task & 31, tk = (task >> 5) % T, tj = (task >> 5) / T;
    const int c0 = tj * 16 + (lane >> 2), k0 = tk * 16 + 2 * (lane & 3);
    double2 v[8];
    int e[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int c = c0 + 8 * (k >> 2), r = k0 + (k & 1) + 8 * ((k >> 1) & 1);
      v[k] = r < M && c < M ? getB(r, c) : make_double2(0.0, 0.0);
      e[k] = c < M ? eb[c] : 0;
    }
    write_residues(v, e, dig + ((int64_t)tj * T + tk) * 32 + lane, plane);
  }
}

// A CTA of 8 warps computes a 64 x 64 block: warps 0..3 the u products of its
// four 32 x 32 quadrants, warps 4..7 the v products.  The planes of 32 k (16
// KB: 4 row and 4 column tiles, u and v) are staged in shared memory with
// cp.async, kStages deep (stg: kStageUint4), the moduli in sequence; with two
// stages of 64 k instead the copies' latency left a step at 2,800 clocks for
// 550 of mma.sync.
constexpr int kBlkTiles = 4;
constexpr int kStageK = 2;                                   // k tiles of a stage
constexpr int kOneUint4 = 2 * 2 * kBlkTiles * kStageK * 32;  // [A, B][u, v][tile][k tile][lane]
constexpr int kStages = 4;
constexpr int kStageUint4 = kStages * kOneUint4;

// Stores C_ij by out(i, j, re, im) for i, j < M in the block at tiles (ti0,
// tj0); res: the CTA's scratch (kBlockUint4).
template <class Out>
__device__ void gemm_block(int M, int ti0, int tj0, const uint4* adig, const uint4* bdig, const int* ea, const int* eb,
                           uint4* stg, uint4* res, Out out) {
  const int T = oz::tiles(M);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int uv = warp >> 2, quad = warp & 3, qr = quad >> 1, qc = quad & 1;
  const int64_t plane = (int64_t)T * T * 32;
  const int nch = (T + kStageK - 1) / kStageK;  // stages of a modulus
  const int nsteps = kMod * nch;
  // The 4 copies of a thread and step: element e of the stage is lane e & 31
  // of k tile (e >> 5) & 1 of tile (e >> 6) & 3 of plane (e >> 8) & 1 of A
  // (e < 512) or B; the addresses advance by stage and modulus.
  const uint4* src[4];
  bool on[4];
  const int kt0 = (tid >> 5) & 1;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int e = tid + 256 * q;
    const int tile = (e >> 6) & 3, pl = (e >> 8) & 1;
    const int t = (q >= 2 ? tj0 : ti0) + tile;
    on[q] = t < T;
    src[q] = (q >= 2 ? bdig : adig) + pl * plane + ((int64_t)t * T + kt0) * 32 + (e & 31);
  }
  int fm = 0, fch = 0;  // modulus and stage of the next fetch
  auto fetch = [&](int step) {
    if (step < nsteps) {
      uint4* dst = stg + (step % kStages) * kOneUint4;
      const int64_t off = 2 * fm * plane + fch * (kStageK * 32);
      const bool kin = fch * kStageK + kt0 < T;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (on[q] && kin) oz::cp_async16(dst + tid + 256 * q, src[q] + off);
      if (++fch == nch) {
        fch = 0;
        ++fm;
      }
    }
    oz::cp_async_commit();
  };
  float acc[2][2][8];
  __syncthreads();  // the stages' previous contents have been used
  for (int k = 0; k < kStages - 1; ++k) fetch(k);
  int m = 0, ch = 0;
  for (int step = 0; step < nsteps; ++step) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();  // this stage is here, and the one before it has been used
    fetch(step + kStages - 1);
    if (ch == 0) {
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int w = 0; w < 8; ++w) acc[i][j][w] = 0.0f;
    }
    const uint4* cur = stg + (step % kStages) * kOneUint4;
    const uint4* As = cur + (uv * 4 + 2 * qr) * (kStageK * 32) + lane;
    const uint4* Bs = cur + 512 + (uv * 4 + 2 * qc) * (kStageK * 32) + lane;
    const int nk = min(kStageK, T - kStageK * ch);
#pragma unroll
    for (int kt = 0; kt < kStageK; ++kt) {
      if (kt < nk) {
        uint4 af[2], bf[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          af[i] = As[(i * kStageK + kt) * 32];
          bf[i] = Bs[(i * kStageK + kt) * 32];
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            oz::mma16816(acc[i][j], af[i], bf[j].x, bf[j].y);
            oz::mma16816(acc[i][j] + 4, af[i], bf[j].z, bf[j].w);
          }
      }
    }
    const bool last = ch == nch - 1;
    if (last || (ch & 1)) {  // 64 k at most since the last reduction
      const float p = kT.p[m], inv = kT.inv[m];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int w = 0; w < 8; ++w) acc[i][j][w] = reduce(acc[i][j][w], p, inv);
    }
    if (last) {
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float* a = acc[i][j];
          __stcg(res + ((2 * m + uv) * 16 + quad * 4 + 2 * i + j) * 32 + lane,
                 make_uint4(pack_half2(a[0], a[1]), pack_half2(a[2], a[3]), pack_half2(a[4], a[5]),
                            pack_half2(a[6], a[7])));
        }
      ++m;
      ch = 0;
    } else {
      ++ch;
    }
  }
  __syncthreads();  // the residues are written
  // Chinese remainders, four entries of one n8 tile at a time.
  const int g = lane >> 2, t4 = lane & 3;
#pragma unroll 1
  for (int task = warp; task < 32; task += 8) {
    const int n = task & 1, j = (task >> 1) & 1, i = (task >> 2) & 1, qd = task >> 3;
    const int ti = ti0 + 2 * (qd >> 1) + i, tj = tj0 + 2 * (qd & 1) + j;
    if (ti >= T || tj >= T) continue;
    const uint2* src = reinterpret_cast<const uint2*>(res + (qd * 4 + 2 * i + j) * 32 + lane) + n;
    unsigned long long s0[8], s1[8], s2[8];  // re of the four entries, then im
    float2 kf[4];
#pragma unroll
    for (int w = 0; w < 8; ++w) s0[w] = s1[w] = s2[w] = 0ULL;
#pragma unroll
    for (int w = 0; w < 4; ++w) kf[w] = make_float2(0.0f, 0.0f);
    // the residues of four moduli are loaded while those of the last four are used
    uint2 U[4], V[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      U[q] = __ldcg(src + (2 * q) * 1024);
      V[q] = __ldcg(src + (2 * q + 1) * 1024);
    }
#pragma unroll 1
    for (int m0 = 0; m0 < kMod; m0 += 4) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int mm = m0 + q;
        const uint2 Uq = U[q], Vq = V[q];
        if (mm + 4 < kMod) {
          U[q] = __ldcg(src + (2 * (mm + 4)) * 1024);
          V[q] = __ldcg(src + (2 * (mm + 4) + 1) * 1024);
        }
        const float2 mp = both(-kT.p[mm]), inv = both(kT.inv[mm]);
        const uint32_t g0 = kT.g[mm][0], g1 = kT.g[mm][1], g2 = kT.g[mm][2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          __half2 uh, vh;
          const uint32_t uw = h ? Uq.y : Uq.x, vw = h ? Vq.y : Vq.x;
          memcpy(&uh, &uw, 4);
          memcpy(&vh, &vw, 4);
          const float2 u = __half22float2(uh), v = __half22float2(vh);
          const float2 x[2] = {mul2(add2(u, v), both(kT.k1[mm])), mul2(fma2(v, both(-1.0f), u), both(kT.k2[mm]))};
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const float2 r = reduce2(x[c], mp, inv);
            kf[2 * c + h] = fma2(r, inv, kf[2 * c + h]);
            const float2 am = add2(r, both(kMagic + 1024.0f));  // r + 1024 in the low bits
            const uint32_t a0 = __float_as_uint(am.x) & 4095u, a1 = __float_as_uint(am.y) & 4095u;
            const int w = 4 * c + 2 * h;
            s0[w] += (unsigned long long)a0 * g0;
            s1[w] += (unsigned long long)a0 * g1;
            s2[w] += (unsigned long long)a0 * g2;
            s0[w + 1] += (unsigned long long)a1 * g0;
            s1[w + 1] += (unsigned long long)a1 * g1;
            s2[w + 1] += (unsigned long long)a1 * g2;
          }
        }
      }
    }
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const int row = ti * 16 + g + ((w & 2) ? 8 : 0), col = tj * 16 + n * 8 + 2 * t4 + (w & 1);
      if (row < M && col < M) {
        const int e = ea[row] + eb[col] - 106 + kUnit;
        double r[2];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int x = 4 * c + w;
          // s - off - k q modulo 2^96, as hi64 : lo32
          const long long k = (long long)__float2int_rn((x & 1) ? kf[x >> 1].y : kf[x >> 1].x);
          const unsigned long long t0 = s0[x] - (unsigned long long)kT.off[0];
          const unsigned long long kq0 = (unsigned long long)(k * (long long)kT.q[0]);
          const unsigned long long kq1 = (unsigned long long)(k * (long long)kT.q[1]);
          const unsigned long long kq2 = (unsigned long long)(k * (long long)kT.q[2]);
          const unsigned long long l0 = t0 - kq0;  // signed, |l0| < 2^49
          const unsigned long long l1 = s1[x] - kT.off[1] - kq1 + (unsigned long long)((long long)l0 >> 32);
          const unsigned long long l2 = s2[x] - kT.off[2] - kq2 + (unsigned long long)((long long)l1 >> 32);
          const long long top = (long long)((l2 << 32) | (l1 & 0xffffffffULL));  // bits 32..95
          const uint32_t low = (uint32_t)l0;
          const int sh = min(32, __clzll(top < 0 ? ~top : top) - 2);
          r[c] = oz::fix_to_double((top << sh) + (long long)((unsigned long long)low >> (32 - sh)), e + 32 - sh);
        }
        out(row, col, r[0], r[1]);
      }
    }
  }
}

}  // namespace crt
}  // namespace rg
