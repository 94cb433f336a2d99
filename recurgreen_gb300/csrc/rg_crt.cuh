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
//  * the residues of an integer are its six 9-bit limbs times constants modulo
//    p, one mma for 16 planes and 8 entries (split);
//  * residues are balanced, |r| <= 511, exact in FP16; sums over 64 k stay
//    below 64 511^2 + 511 < 2^24, so they are exact in FP32, and are reduced
//    modulo p after every 64 k;
//  * C'/P = sum_m (u_m + v_m) k_m / p_m modulo 1 with constants k_m (for the
//    imaginary part u_m - v_m), |C'| < P/8: the fractions k_m / p_m, to 88
//    bits in balanced base-2^11 digits, are again an mma's other operand, whose
//    eight sums (below 2^24, exact) make up C'/P modulo 1 in integers.  The
//    rounding of the fractions is below 2^44 in C' (the operands' own rounding
//    is near 2^56); the result is rounded to FP64 once.
//
// The result depends on neither tiling nor order.  What it replaces in the
// blocked sweep is the digit loop (oz::gemm_block): 7.5k clocks per 32 x 64
// block and 16 k with two CTAs on an SM, bound by instructions around the mma
// (1,400 a warp for 208), the folds of the level sums above all.
//
// Layout: an operand's planes are uint4 [12 moduli][u, v][T tiles along rows
// (A) or columns (B)][T k tiles][32 lanes], in the order of the A fragments of
// A or of B^T: the planes of one serve as the other's.
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>

#include "rg_ozaki.cuh"

namespace rg {
namespace crt {

constexpr int kMod = 12;
constexpr int kFracBits = 88;  // of C'/P: eight balanced digits of 11 bits

__host__ __device__ inline int64_t operand_uint4(int M) {
  const int64_t T = oz::tiles(M);
  return 2LL * kMod * T * T * 32;
}
// Scratch of one CTA for the residues of a 64 x 64 block, in uint4.
constexpr int64_t kBlockUint4 = 2LL * kMod * 16 * 32;

struct Tables {
  float p[kMod], inv[kMod];  // modulus and its reciprocal
  // Fragments by lane (g, t), pairs of FP16 integers.  Limbs to residues (A
  // operand, rows = planes 2 m + v; column of the limbs: lane t has limbs 0, 1,
  // 2 of the 27-bit half t & 1 of the part t >> 1): planes g and g + 8 of limbs
  // 0, 1; of limb 2; plane g + 16 of limbs 0, 1; of limb 2.
  uint32_t split[32][6];
  // Residues to digits of C'/P (B operand, column g = digit g): moduli 2 t, 2 t
  // + 1 and 2 t + 8, 2 t + 9 for the real part, then for the imaginary part.
  uint32_t join[32][4];
  long long top;  // P in kTopBits bits
  int shift;      // and P = top 2^shift
};
constexpr int kTopBits = 63;

typedef unsigned __int128 u128;
typedef __int128 i128;

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

constexpr uint32_t half_of(int x) {  // FP16 bits of an integer, |x| <= 2048
  if (x == 0) return 0;
  uint32_t a = (uint32_t)(x < 0 ? -x : x), e = 25;
  while (a < 1024) a <<= 1, --e;
  if (a >= 2048) a >>= 1, ++e;  // (2048 itself)
  return (x < 0 ? 0x8000u : 0u) | (e << 10) | (a & 1023u);
}
constexpr uint32_t half_pair(int a, int b) { return half_of(a) | half_of(b) << 16; }

constexpr Tables make_tables() {
  Tables t{};
  u128 P = 1;
  for (int m = 0; m < kMod; ++m) P *= (u128)kModuli[m];
  int digits[2][kMod][8] = {};
  for (int m = 0; m < kMod; ++m) {
    const int p = kModuli[m];
    const int inv = inverse((int)(P / (u128)p % (u128)p), p), s = root_of_minus_one(p);
    t.p[m] = (float)p;
    t.inv[m] = 1.0f / (float)p;
    for (int c = 0; c < 2; ++c) {  // C'_re: (u + v)/2, C'_im: (u - v)/(2 s)
      const int k = balanced((long long)inv * inverse(c ? 2 * s : 2, p), p);
      i128 f = (i128)k * ((i128)1 << kFracBits) * 2;
      f = (f + (f < 0 ? -p : p)) / (2 * p);
      for (int d = 0; d < 8; ++d) {
        const int r = d < 7 ? (int)(((f + 1024) & 2047) - 1024) : (int)f;
        digits[c][m][d] = r;
        f = (f - r) / 2048;
      }
    }
  }
  for (int lane = 0; lane < 32; ++lane) {
    const int g = lane >> 2, q = lane & 3;
    for (int w = 0; w < 3; ++w) {
      const int plane = g + 8 * w, p = kModuli[plane >> 1], s = root_of_minus_one(p);
      int c[3] = {};
      for (int j = 0; j < 3; ++j) {
        long long x = (1LL << (9 * j + 27 * (q & 1))) % p;
        if (q >> 1) x = x * ((plane & 1) ? p - s : s) % p;
        c[j] = balanced(x, p);
      }
      t.split[lane][w < 2 ? w : 4] = half_pair(c[0], c[1]);
      t.split[lane][w < 2 ? w + 2 : 5] = half_pair(c[2], 0);
    }
    for (int c = 0; c < 2; ++c) {
      t.join[lane][2 * c] = half_pair(digits[c][2 * q][g], digits[c][2 * q + 1][g]);
      t.join[lane][2 * c + 1] = q < 2 ? half_pair(digits[c][2 * q + 8][g], digits[c][2 * q + 9][g]) : 0;
    }
  }
  while ((P >> (t.shift + kTopBits)) != 0) ++t.shift;
  t.top = (long long)(P >> t.shift);
  return t;
}
static __device__ const Tables kT = make_tables();

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
__device__ __forceinline__ float2 both(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 reduce2(float2 x, float2 mp, float2 inv) {  // mp = -p
  const float2 q = add2(fma2(x, inv, both(kMagic)), both(-kMagic));
  return fma2(q, mp, x);
}

__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  uint32_t r;
  memcpy(&r, &h, 4);
  return r;
}

__device__ __forceinline__ uint32_t sub_half2(uint32_t a, uint32_t b) {
  __half2 x, y;
  memcpy(&x, &a, 4);
  memcpy(&y, &b, 4);
  x = __hsub2(x, y);
  memcpy(&a, &x, 4);
  return a;
}
__device__ __forceinline__ uint32_t add_half2(uint32_t a, uint32_t b) {
  __half2 x, y;
  memcpy(&x, &a, 4);
  memcpy(&y, &b, 4);
  x = __hadd2(x, y);
  memcpy(&a, &x, 4);
  return a;
}

// Residue planes of an operand with rows i = rows of A or columns of B:
// entries get(i, k) (zero outside M x M), exponents ex[i].  A warp per 16 x 16
// tile, tiles warp0, warp0 + nwarps, ...; stg: kSplitUint4 of shared memory for
// each warp of the CTA.  The entries' integers pass through shared memory, so
// that loads and conversions are made once, and a quad of lanes then has the
// 27-bit halves of both parts of an entry, three limbs a lane.  Residues by
// FP32 multiply-adds instead, 18 and 2 roundings for two entries and a modulus,
// made this phase as long as the product itself at 256 modes.
constexpr int kSplitUint4 = 32 * 10;  // a lane's 8 entries, and 32 bytes against bank conflicts
template <class Get>
__device__ __forceinline__ void split(int M, Get get, const int* ex, uint4* dig, uint4* stg, int warp0, int nwarps) {
  const int T = oz::tiles(M), lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int64_t plane = (int64_t)T * T * 32;
  uint4* st = stg + (threadIdx.x >> 5) * kSplitUint4;
  const uint32_t* sw = reinterpret_cast<const uint32_t*>(st) + (g >> 1) * 40 + (g & 1) * 4 + t;
  uint32_t wt[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) wt[k] = kT.split[lane][k];
  float2 mp[3], inv[3];
#pragma unroll
  for (int w = 0; w < 3; ++w) {
    mp[w] = both(-kT.p[(g >> 1) + 4 * w]);
    inv[w] = both(kT.inv[(g >> 1) + 4 * w]);
  }
  for (int tile = warp0; tile < T * T; tile += nwarps) {
    const int tk = tile % T, ti = tile / T;
    const int r0 = ti * 16 + g, k0 = tk * 16 + 2 * t;
    __syncwarp();  // the last tile's integers have been used
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int r = r0 + 8 * ((k >> 1) & 1), c = k0 + (k & 1) + 8 * (k >> 2);
      const double2 v = r < M && c < M ? get(r, c) : make_double2(0.0, 0.0);
      const int e = r < M ? ex[r] : 0;
      const long long x = oz::sfixed53(v.x, e), y = oz::sfixed53(v.y, e);
      st[lane * 10 + k] = make_uint4((uint32_t)x & 0x7ffffffu, (uint32_t)(x >> 27), (uint32_t)y & 0x7ffffffu,
                                     (uint32_t)(y >> 27));
    }
    __syncwarp();
    uint4* dst = dig + (int64_t)tile * 32 + g * plane + t;
#pragma unroll 2
    for (int grp = 0; grp < 8; ++grp) {  // entries of lanes 4 grp .. 4 grp + 3
      uint32_t out[3][4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t x = sw[grp * 160 + q * 8];
        // limbs as FP16: 1024 + l has l in its low bits; the last is signed
        const uint32_t l01 = (x & 511u) | ((x & 0x3fe00u) << 7) | 0x64006400u;
        const uint32_t l2 = (uint32_t)(((int)x >> 18) + 512) | 0x64006400u;
        const uint32_t b0 = sub_half2(l01, 0x64006400u), b1 = sub_half2(l2, 0x64006600u);
        float c[4] = {0.0f, 0.0f, 0.0f, 0.0f}, d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        oz::mma16816(c, make_uint4(wt[0], wt[1], wt[2], wt[3]), b0, b1);
        oz::mma16816(d, make_uint4(wt[4], 0u, wt[5], 0u), b0, b1);
        const float2 u0 = reduce2(make_float2(c[0], c[1]), mp[0], inv[0]);
        const float2 u1 = reduce2(make_float2(c[2], c[3]), mp[1], inv[1]);
        const float2 u2 = reduce2(make_float2(d[0], d[1]), mp[2], inv[2]);
        out[0][q] = pack_half2(u0.x, u0.y);
        out[1][q] = pack_half2(u1.x, u1.y);
        out[2][q] = pack_half2(u2.x, u2.y);
      }
#pragma unroll
      for (int w = 0; w < 3; ++w)
        __stcg(dst + 8 * w * plane + 4 * grp, make_uint4(out[w][0], out[w][1], out[w][2], out[w][3]));
    }
  }
}

// A CTA of 8 warps computes a 64 x 64 block: warps 0..3 the u products of its
// four 32 x 32 quadrants, warps 4..7 the v products.  The planes of 64 k (32
// KB: 4 row and 4 column tiles, u and v) are staged in shared memory with
// cp.async, kStages deep (stg: kStageUint4), the moduli in sequence; the sums
// of a stage stay exact, and are reduced modulo p at its end.  (Four stages of
// 32 k: 126 for 116 ms of 512 modes, t of 16 realizations and 16 slices; 217 for
// 212 ms of 152 at 256 modes.)
constexpr int kBlkTiles = 4;
constexpr int kStageK = 4;                                        // k tiles of a stage
constexpr int kHalfUint4 = 2 * kBlkTiles * kStageK * 32;          // [u, v][tile][k tile][lane]
constexpr int kOneUint4 = 2 * kHalfUint4;                         // of A, then of B
constexpr int kStages = 3;
constexpr int kStageUint4 = kStages * kOneUint4;

// Stores C_ij by out(i, j, 0, re) and out(i, j, 1, im) for i, j < M in the
// block at tiles (ti0, tj0); res: the CTA's scratch (kBlockUint4).
template <class Out>
__device__ void gemm_block(int M, int ti0, int tj0, const uint4* adig, const uint4* bdig, const int* ea, const int* eb,
                           uint4* stg, uint4* res, Out out) {
  const int T = oz::tiles(M);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int uv = warp >> 2, quad = warp & 3, qr = quad >> 1, qc = quad & 1;
  const int64_t plane = (int64_t)T * T * 32;
  const int nch = (T + kStageK - 1) / kStageK;  // stages of a modulus
  const int nsteps = kMod * nch;
  // The 8 copies of a thread and step: element e = tid + 256 q of the stage is
  // lane e & 31 of k tile (e >> 5) & 3 of tile (e >> 7) & 3 of plane (e >> 9) &
  // 1 of A (e < 1024) or B.
  const int kt0 = (tid >> 5) & 3, tl0 = tid >> 7;  // tiles tl0 and tl0 + 2
  const int64_t at = ((int64_t)tl0 * T + kt0) * 32 + lane;
  const uint4* asrc = adig + (int64_t)ti0 * T * 32 + at;
  const uint4* bsrc = bdig + (int64_t)tj0 * T * 32 + at;
  const int two = 2 * T * 32;  // two tiles on
  const bool a0 = ti0 + tl0 < T, a1 = ti0 + tl0 + 2 < T, b0 = tj0 + tl0 < T, b1 = tj0 + tl0 + 2 < T;
  int fm = 0, fch = 0;  // modulus and stage of the next fetch
  auto fetch = [&](int step) {
    if (step < nsteps) {
      uint4* dst = stg + (step % kStages) * kOneUint4 + tid;
      if (fch * kStageK + kt0 < T) {
        const int64_t off = 2 * fm * plane + fch * (kStageK * 32);
#pragma unroll
        for (int pl = 0; pl < 2; ++pl) {
          if (a0) oz::cp_async16(dst + 512 * pl, asrc + off + pl * plane);
          if (a1) oz::cp_async16(dst + 512 * pl + 256, asrc + off + pl * plane + two);
          if (b0) oz::cp_async16(dst + kHalfUint4 + 512 * pl, bsrc + off + pl * plane);
          if (b1) oz::cp_async16(dst + kHalfUint4 + 512 * pl + 256, bsrc + off + pl * plane + two);
        }
      }
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
    const float2 mp = both(-kT.p[m]), inv = both(kT.inv[m]);
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
    const uint4* Bs = cur + kHalfUint4 + (uv * 4 + 2 * qc) * (kStageK * 32) + lane;
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
            oz::mma16816(acc[i][j], af[i], bf[j].x, bf[j].z);
            oz::mma16816(acc[i][j] + 4, af[i], bf[j].y, bf[j].w);
          }
      }
    }
    const bool last = ch == nch - 1;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int w = 0; w < 8; w += 2) {
          const float2 r = reduce2(make_float2(acc[i][j][w], acc[i][j][w + 1]), mp, inv);
          acc[i][j][w] = r.x;
          acc[i][j][w + 1] = r.y;
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
  // Chinese remainders.  A lane takes the words of lane 8 h + g of a tile, for
  // moduli 2 t, 2 t + 1 and 2 t + 8, 2 t + 9: row g of an mma is a word's first
  // entry, row g + 8 its second.  Its sums, two digits of four numbers (two
  // entries, re and im), go through shared memory, and lane t of a quad ends
  // up with all digits of number t.
  const int g = lane >> 2, t4 = lane & 3;
  long long* part = reinterpret_cast<long long*>(stg) + (warp * 8 + g) * 18;  // [4 numbers][4], two against conflicts
  uint32_t jc[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) jc[k] = kT.join[lane][k];
#pragma unroll 1
  for (int task = warp; task < 64; task += 8) {
    const int h = task & 3, i = (task >> 3) & 1, j = (task >> 2) & 1, qd = task >> 4;
    const int ti = ti0 + 2 * (qd >> 1) + i, tj = tj0 + 2 * (qd & 1) + j;
    if (ti >= T || tj >= T) continue;
    const uint4* src = res + (qd * 4 + 2 * i + j) * 32 + 8 * h + g;
    uint4 re[4], im[4];  // sums and differences of u and v for the four moduli
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      re[k] = im[k] = make_uint4(0u, 0u, 0u, 0u);
      const int mm = 2 * t4 + (k & 1) + 8 * (k >> 1);
      if (mm < kMod) {
        const uint4 u = __ldcg(src + (2 * mm) * 512), v = __ldcg(src + (2 * mm + 1) * 512);
        re[k] = make_uint4(add_half2(u.x, v.x), add_half2(u.y, v.y), add_half2(u.z, v.z), add_half2(u.w, v.w));
        im[k] = make_uint4(sub_half2(u.x, v.x), sub_half2(u.y, v.y), sub_half2(u.z, v.z), sub_half2(u.w, v.w));
      }
    }
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      auto word = [&](const uint4& x) { return w == 0 ? x.x : w == 1 ? x.y : w == 2 ? x.z : x.w; };
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const uint4* x = c ? im : re;
        const uint32_t x0 = word(x[0]), x1 = word(x[1]), x2 = word(x[2]), x3 = word(x[3]);
        float d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        oz::mma16816(d, make_uint4(__byte_perm(x0, x1, 0x5410), __byte_perm(x0, x1, 0x7632),
                                   __byte_perm(x2, x3, 0x5410), __byte_perm(x2, x3, 0x7632)),
                     jc[2 * c], jc[2 * c + 1]);
        part[c * 4 + t4] = (long long)__float2int_rn(d[0]) + (long long)__float2int_rn(d[1]) * 2048;
        part[(2 + c) * 4 + t4] = (long long)__float2int_rn(d[2]) + (long long)__float2int_rn(d[3]) * 2048;
      }
      __syncwarp();
      const longlong2 p01 = *reinterpret_cast<const longlong2*>(part + t4 * 4);
      const longlong2 p23 = *reinterpret_cast<const longlong2*>(part + t4 * 4 + 2);
      __syncwarp();
      const int row = ti * 16 + 2 * h + (g >> 2) + 8 * (w & 1);
      const int col = tj * 16 + 8 * (w >> 1) + 2 * (g & 3) + (t4 >> 1);
      if (row < M && col < M) {
        // C'/P 2^88 = lo + 2^44 hi modulo 2^88: its top 64 bits, and 24 more
        const long long lo = p01.x + p01.y * (1LL << 22);
        const unsigned long long hi =
            (unsigned long long)p23.x + ((unsigned long long)p23.y << 22) + (unsigned long long)(lo >> 44);
        const long long top = (long long)((hi << 20) | (unsigned)((lo >> 24) & 0xfffff));
        const unsigned rest = (unsigned)lo & 0xffffffu;
        const int sh = min(24, __clzll(top < 0 ? ~top : top) - 1);
        const long long f = (long long)((unsigned long long)top << sh) + (long long)(rest >> (24 - sh));
        out(row, col, t4 & 1,
            oz::fix_to_double(__mul64hi(f, kT.top), ea[row] + eb[col] - 106 + kT.shift - sh));
      }
    }
  }
}

}  // namespace crt
}  // namespace rg
