// Complex FP64 matrix products on the FP16 tensor cores (Ozaki splitting).
//
// C = A B for M x M complex matrices (M <= 512), computed with mma.sync
// m16n8k16 (FP16 inputs, FP32 accumulation) to FP64 accuracy:
//
//  * every row i of A gets the exponent ea_i of its largest |re| or |im|
//    (|A_ik| < 2^ea_i), every column j of B the exponent eb_j likewise;
//  * each entry is written as a 53-bit fixed-point integer relative to that
//    power of two (rounded to nearest), X = |A_ik| 2^(53-ea_i) < 2^53, and
//    cut into six balanced base-512 digits (from the least significant up,
//    a digit of 256 or more becomes digit - 512 with a carry into the next;
//    the top one takes the last carry), so |d_p| <= 256 and
//        A_ik = 2^ea_i sum_p d_p 2^(-8-9p),  p = 0..5
//    (each digit exact in FP16, each product of two below 2^16);
//  * C_ij = 2^(ea_i + eb_j) sum_l v_l 2^(-16-9l) with
//        v_l = sum_{p+q=l} sum_k a_p(i,k) b_q(k,j),
//    and levels l <= 6 kept (26 digit pairs; the first dropped level lies
//    near 2^-53 K relative to 2^(ea_i+eb_j), an FP64 product's own error
//    bound);
//  * v_l is accumulated in FP32 over chunks of 16 complex k: at most
//    6 pairs x 32 real products x 2^16 = 12,582,912 < 2^24 per level, so
//    every partial sum is an integer below 2^24 and the accumulation is
//    exact; after each chunk the levels are folded into two int64 sums,
//    hi = sum_{l<=2} v_l 2^(9(2-l)) and lo = sum_{l>=3} v_l 2^(9(6-l)),
//    which are exact too (|hi| < 2^46, |lo| < 2^56 for M <= 512);
//  * finally C_ij = 2^(ea_i+eb_j) (hi 2^-34 + lo 2^-70), one rounding.
//
// The result is the correctly rounded value of the digit sum, so it does
// not depend on how tiles are spread over warps or CTAs, and it equals an
// exact integer model of the same steps bit for bit.  Its error is that of
// the dropped digit pairs and the 2^-53 rounding of the inputs, i.e.
// normwise at the level of an FP64 product (2^-53 K |A_i| |B_j| at worst).
//
// Layouts ("fragment-native", so a lane loads its mma operand with one
// 16-byte access).  With T = ceil(M/16) tiles per dimension:
//   A digits  uint4 [2 parts][6 slices][T row tiles][T k tiles][32 lanes]
//             lane (g = lane/4, t = lane%4) of tile (ti, tk) holds the halves
//             (A[g][2t], A[g][2t+1]), (A[g+8][2t], A[g+8][2t+1]),
//             (A[g][2t+8], A[g][2t+9]), (A[g+8][2t+8], A[g+8][2t+9])
//             of the 16 x 16 tile: the m16n8k16 A fragment (row-major);
//   B digits  uint4 [2 parts][6 slices][T col tiles][T k tiles][32 lanes]
//             lane holds (B[2t][g], B[2t+1][g]), (B[2t+8][g], B[2t+9][g]) of
//             columns 0..7 of the tile, then the same for columns 8..15: two
//             m16n8k16 B fragments (column-major);
//   accumulators: c0 = C[g][2t], c1 = C[g][2t+1], c2 = C[g+8][2t], c3 = C[g+8][2t+1].
// Rows/columns beyond M are zero digits.
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>

namespace rg {
namespace oz {

constexpr int kSlices = 6;      // digits per entry
constexpr int kDigitBits = 9;   // base 2^9, balanced digits in [-256, 256]
constexpr int kFixedBits = 53;  // fixed-point bits of an entry
constexpr int kLmax = 6;        // highest level kept
constexpr int kHiLevels = 3;    // levels 0..2 fold into hi, 3..6 into lo
constexpr int kNoExp = -4096;   // exponent of zero rows
// C = 2^(ea+eb) (hi kHiScale + lo kLoScale)
constexpr double kHiScale = 0x1p-34;  // 2^-(16 + 9 (kHiLevels - 1))
constexpr double kLoScale = 0x1p-70;  // 2^-(16 + 9 kLmax)

__host__ __device__ inline int tiles(int M) { return (M + 15) >> 4; }
// uint4 elements of one operand's digits
__host__ __device__ inline int64_t operand_uint4(int M) {
  const int64_t T = tiles(M);
  return 2LL * kSlices * T * T * 32;
}
// bytes of both operands' digits plus the exponents (2 x M ints, 16-byte padded)
__host__ __device__ inline int64_t workspace_bytes(int M) {
  return 2 * 16 * operand_uint4(M) + (((int64_t)2 * tiles(M) * 16 * 4 + 15) & ~15LL);
}

// frexp exponent of |x| (|x| < 2^e), kNoExp for zeros and subnormals.
__device__ __forceinline__ int fexp(double x) {
  const int eb = (int)((__double_as_longlong(x) >> 52) & 0x7ff);
  return eb == 0 ? kNoExp : eb - 1022;
}

__device__ __forceinline__ int fexp2(double2 v) { return max(fexp(v.x), fexp(v.y)); }

// |x| 2^(53-e) rounded to nearest, as an integer below 2^53 (e >= fexp(x)).
__device__ __forceinline__ uint64_t fixed53(double x, int e) {
  const uint64_t bits = (uint64_t)__double_as_longlong(x);
  const int eb = (int)((bits >> 52) & 0x7ff);
  if (eb == 0) return 0;
  const uint64_t m = (bits & ((1ULL << 52) - 1)) | (1ULL << 52);
  const int rs = e - (eb - 1022);  // |x| 2^(53-e) = m 2^-rs, rs >= 0
  if (rs == 0) return m;
  if (rs > 54) return 0;
  return (m + (1ULL << (rs - 1))) >> rs;
}

// The six balanced base-512 digits of X < 2^53, d[0] the most significant:
// X = sum_p d[p] 2^(9(5-p)), |d[p]| <= 256.
__device__ __forceinline__ void balanced_digits(uint64_t X, int d[kSlices]) {
  int carry = 0;
#pragma unroll
  for (int p = kSlices - 1; p > 0; --p) {
    const int t = (int)((X >> (kDigitBits * (kSlices - 1 - p))) & 511u) + carry;
    carry = t >= 256 ? 1 : 0;
    d[p] = t - (carry << 9);
  }
  d[0] = (int)(X >> (kDigitBits * (kSlices - 1))) + carry;
}

// Two signed digits as FP16 halves (lo = first); the entries' signs n0, n1
// multiply them.  A magnitude m <= 256 is made exact in FP16 as
// (1024 + m) - 1024, then the sign bit is set.
__device__ __forceinline__ uint32_t digit_pair(int d0, bool n0, int d1, bool n1) {
  const uint32_t m0 = (uint32_t)abs(d0), m1 = (uint32_t)abs(d1);
  const uint32_t biased = (0x6400u | m0) | ((0x6400u | m1) << 16);
  __half2 h;
  memcpy(&h, &biased, 4);
  h = __hsub2(h, __floats2half2_rn(1024.0f, 1024.0f));
  uint32_t r;
  memcpy(&r, &h, 4);
  // the sign of a zero digit does not matter (its products are +-0)
  return r ^ ((n0 != (d0 < 0) ? 0x8000u : 0u) | (n1 != (d1 < 0) ? 0x80000000u : 0u));
}

// Writes the 12 uint4 (2 parts x 6 slices) of one lane of one tile from its
// 8 complex entries v[0..7] in fragment order (see the layout above) and
// the row (A) or column (B) exponents of each entry: for A, entries 0,1,4,5
// lie on row g and 2,3,6,7 on row g+8; for B, entries 0..3 on column g and
// 4..7 on column g+8.  dst points at [part 0][slice 0][this tile][lane];
// `plane` is the uint4 stride between slices.
__device__ __forceinline__ void write_digits(const double2 v[8], const int e[8], uint4* dst, int64_t plane) {
  uint32_t rw[kSlices][4], iw[kSlices][4];
#pragma unroll
  for (int w = 0; w < 4; ++w) {
    int dr0[kSlices], dr1[kSlices], di0[kSlices], di1[kSlices];
    balanced_digits(fixed53(v[2 * w].x, e[2 * w]), dr0);
    balanced_digits(fixed53(v[2 * w + 1].x, e[2 * w + 1]), dr1);
    balanced_digits(fixed53(v[2 * w].y, e[2 * w]), di0);
    balanced_digits(fixed53(v[2 * w + 1].y, e[2 * w + 1]), di1);
#pragma unroll
    for (int p = 0; p < kSlices; ++p) {
      rw[p][w] = digit_pair(dr0[p], v[2 * w].x < 0.0, dr1[p], v[2 * w + 1].x < 0.0);
      iw[p][w] = digit_pair(di0[p], v[2 * w].y < 0.0, di1[p], v[2 * w + 1].y < 0.0);
    }
  }
#pragma unroll
  for (int p = 0; p < kSlices; ++p) {
    __stcg(dst + p * plane, make_uint4(rw[p][0], rw[p][1], rw[p][2], rw[p][3]));
    __stcg(dst + (kSlices + p) * plane, make_uint4(iw[p][0], iw[p][1], iw[p][2], iw[p][3]));
  }
}

// Digit planes of A: entries A(i, k) = getA(i, k) (zero outside M x M),
// exponents ea[i].  Task = (row tile, k tile, lane), spread over
// [task0, ntask) with stride `step`.
template <class GetA>
__device__ void split_a(int M, GetA getA, const int* ea, uint4* dig, int task0, int step) {
  const int T = tiles(M);
  const int64_t plane = (int64_t)T * T * 32;
  const int ntask = T * T * 32;
  for (int task = task0; task < ntask; task += step) {
    const int lane = task & 31, tk = (task >> 5) % T, ti = (task >> 5) / T;
    const int g = lane >> 2, t = lane & 3;
    const int r0 = ti * 16 + g, r1 = r0 + 8;
    const int cs[4] = {tk * 16 + 2 * t, tk * 16 + 2 * t + 1, tk * 16 + 2 * t + 8, tk * 16 + 2 * t + 9};
    double2 v[8];
    int e[8];
    const int rows[8] = {r0, r0, r1, r1, r0, r0, r1, r1};
    const int cols[8] = {cs[0], cs[1], cs[0], cs[1], cs[2], cs[3], cs[2], cs[3]};
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const bool in = rows[k] < M && cols[k] < M;
      v[k] = in ? getA(rows[k], cols[k]) : make_double2(0.0, 0.0);
      e[k] = rows[k] < M ? ea[rows[k]] : 0;
    }
    write_digits(v, e, dig + ((int64_t)ti * T + tk) * 32 + lane, plane);
  }
}

// Digit planes of B: entries B(k, j) = getB(k, j), exponents eb[j].
template <class GetB>
__device__ void split_b(int M, GetB getB, const int* eb, uint4* dig, int task0, int step) {
  const int T = tiles(M);
  const int64_t plane = (int64_t)T * T * 32;
  const int ntask = T * T * 32;
  for (int task = task0; task < ntask; task += step) {
    const int lane = task & 31, tk = (task >> 5) % T, tj = (task >> 5) / T;
    const int g = lane >> 2, t = lane & 3;
    const int c0 = tj * 16 + g, c1 = c0 + 8;
    const int ks[4] = {tk * 16 + 2 * t, tk * 16 + 2 * t + 1, tk * 16 + 2 * t + 8, tk * 16 + 2 * t + 9};
    double2 v[8];
    int e[8];
    const int rows[8] = {ks[0], ks[1], ks[2], ks[3], ks[0], ks[1], ks[2], ks[3]};
    const int cols[8] = {c0, c0, c0, c0, c1, c1, c1, c1};
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const bool in = rows[k] < M && cols[k] < M;
      v[k] = in ? getB(rows[k], cols[k]) : make_double2(0.0, 0.0);
      e[k] = cols[k] < M ? eb[cols[k]] : 0;
    }
    write_digits(v, e, dig + ((int64_t)tj * T + tk) * 32 + lane, plane);
  }
}

__device__ __forceinline__ void mma16816(float c[4], const uint4& a, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void cp_async16(uint4* smem_dst, const uint4* gsrc) {
  const unsigned saddr = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(saddr), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
// all but the most recently committed group complete
__device__ __forceinline__ void cp_async_wait_one() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

// ---------------------------------------------------------------------------
// The CTA-blocked product: a CTA of 8 warps computes a 2 x 4 block of 16 x 16
// complex tiles (warp w: row tile ti0 + w/4, column tile tj0 + w%4).  Both
// operands' digits for the block and one k tile -- A for 2 row tiles, B for 4
// column tiles, 36 KB -- are staged in shared memory with cp.async, two
// stages deep (stg: kBlkStageUint4 uint4 = 72 KB), so the copy of k tile
// t + 1 runs while the tensor cores work on k tile t and the loop reads no
// global memory; every staged A digit serves 4 tiles and every B digit 2.
// The level sums of a k tile are folded after it.  out(i, j, re, im) stores C_ij
// (called for i, j < M only).
// ---------------------------------------------------------------------------
constexpr int kBlkRows = 2, kBlkCols = 4;
constexpr int kBlkAUint4 = kBlkRows * 2 * kSlices * 32;                 // one stage's A digits
constexpr int kBlkOneUint4 = (kBlkRows + kBlkCols) * 2 * kSlices * 32;  // one stage
constexpr int kBlkStageUint4 = 2 * kBlkOneUint4;                       // two stages

template <class Out>
__device__ void gemm_block(int M, int ti0, int tj0, const uint4* adig, const uint4* bdig, const int* ea, const int* eb,
                           uint4* stg, Out out) {
  const int T = tiles(M);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wr = warp / kBlkCols, wc = warp % kBlkCols;
  const int ti = ti0 + wr, tj = tj0 + wc;
  const bool active = ti < T && tj < T;
  const int64_t plane = (int64_t)T * T * 32;
  long long hi[16], lo[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) hi[k] = lo[k] = 0;
  // stage element e = (tile * 2 kSlices + part * kSlices + slice) * 32 + lane,
  // the A tiles first, then the B tiles
  auto fetch = [&](int tk, uint4* dst) {
    for (int e = tid; e < kBlkOneUint4; e += blockDim.x) {
      const int isB = e >= kBlkAUint4;
      const int f = isB ? e - kBlkAUint4 : e;
      const int ln = f & 31, ps = (f >> 5) % (2 * kSlices), tile = (f >> 5) / (2 * kSlices);
      const int t = isB ? tj0 + tile : ti0 + tile;
      if (t < T) cp_async16(dst + e, (isB ? bdig : adig) + ps * plane + ((int64_t)t * T + tk) * 32 + ln);
    }
    cp_async_commit();
  };
  __syncthreads();  // the stages' previous contents have been used
  fetch(0, stg);
  for (int tk = 0; tk < T; ++tk) {
    const uint4* cur = stg + (tk & 1) * kBlkOneUint4;
    if (tk + 1 < T) {
      fetch(tk + 1, stg + ((tk + 1) & 1) * kBlkOneUint4);
      cp_async_wait_one();
    } else {
      cp_async_wait_all();
    }
    __syncthreads();  // k tile tk is in `cur` for every warp
    if (active) {
      const uint4* Aw = cur + wr * 2 * kSlices * 32 + lane;
      const uint4* Bw = cur + kBlkAUint4 + wc * 2 * kSlices * 32 + lane;
#pragma unroll 1
      for (int l = 0; l <= kLmax; ++l) {
        float acc[4][4];  // [re n0, re n1, im n0, im n1][4]
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int w = 0; w < 4; ++w) acc[u][w] = 0.0f;
        const int p0 = max(0, l - (kSlices - 1)), p1 = min(l, kSlices - 1);
#pragma unroll 1
        for (int p = p0; p <= p1; ++p) {
          const int q = l - p;
          const uint4 var = Aw[p * 32], vai = Aw[(kSlices + p) * 32];
          const uint4 vb = Bw[q * 32], vc = Bw[(kSlices + q) * 32];
          // re += Ar Br - Ai Bi; im += Ar Bi + Ai Br
          mma16816(acc[0], var, vb.x, vb.y);
          mma16816(acc[0], vai, vc.x ^ 0x80008000u, vc.y ^ 0x80008000u);
          mma16816(acc[1], var, vb.z, vb.w);
          mma16816(acc[1], vai, vc.z ^ 0x80008000u, vc.w ^ 0x80008000u);
          mma16816(acc[2], var, vc.x, vc.y);
          mma16816(acc[2], vai, vb.x, vb.y);
          mma16816(acc[3], var, vc.z, vc.w);
          mma16816(acc[3], vai, vb.z, vb.w);
        }
        const bool in_hi = l < kHiLevels;
        const int sh = in_hi ? kDigitBits * (kHiLevels - 1 - l) : kDigitBits * (kLmax - l);
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int w = 0; w < 4; ++w) {
            const long long v = (long long)__float2int_rn(acc[u][w]) << sh;
            if (in_hi) hi[u * 4 + w] += v;
            else lo[u * 4 + w] += v;
          }
      }
    }
    __syncthreads();  // every warp is done with `cur` before it is refilled
  }
  if (!active) return;
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const int i = ti * 16 + g + ((w & 2) ? 8 : 0);
      const int j = tj * 16 + n * 8 + 2 * t + (w & 1);
      if (i < M && j < M) {
        const int e = ea[i] + eb[j];
        const double re = fma((double)hi[n * 4 + w], kHiScale, (double)lo[n * 4 + w] * kLoScale);
        const double im = fma((double)hi[8 + n * 4 + w], kHiScale, (double)lo[8 + n * 4 + w] * kLoScale);
        out(i, j, scalbn(re, e), scalbn(im, e));
      }
    }
}

// ---------------------------------------------------------------------------
// Products of T x T tiles held in shared memory by one CTA, for the sweep of
// up to 64 modes (rg_sweep_sym.cu).
//
// A plane holds one digit of every entry: [T row tiles][T column tiles][32
// lanes] of 16 bytes, a lane's four words being the A fragment (a0, a1, a2,
// a3) of the layouts above -- which is the accumulator layout of two n8
// tiles, so the owner warp writes its planes from registers.  The same words
// read as a B operand are the transposed tile: (a0, a2) are the fragment of
// columns (= stored rows) 0..7 and (a1, a3) that of 8..15, so these pairs are
// stored together, and swapped in odd octets of lanes: the 8-byte loads of
// one pair are then free of bank conflicts.
// Entries are signed fixed point of 8 + 9 (n - 1) bits, cut into n balanced
// digits in [-256, 255] (the top one up to 256).
// ---------------------------------------------------------------------------

// m 2^-rs rounded to nearest, ties to even (0 < rs < 64).  An entry of half the
// row's largest power of two is a tie every other time: rounded away from zero,
// ties made a slice of the recursion gain 2^-56 (the trace of t^H t + r^H r was
// 1 + 6e-15 after 300 slices of 64 modes, and T off by twice the elimination's
// error).
__device__ __forceinline__ long long shift_even(long long m, int rs) {
  return (m + ((1LL << (rs - 1)) - 1) + ((m >> rs) & 1)) >> rs;
}

// x 2^(53-e) rounded to nearest, ties to even, with sign (|x| < 2^(e+1)).
__device__ __forceinline__ long long sfixed53(double x, int e) {
  const uint64_t bits = (uint64_t)__double_as_longlong(x);
  const int eb = (int)((bits >> 52) & 0x7ff);
  const long long m = (long long)((bits & ((1ULL << 52) - 1)) | (1ULL << 52));
  const int rs = e - (eb - 1022);  // |x| 2^(53-e) = m 2^-rs, rs >= -1
  long long v = rs < 0 ? m << 1 : m;
  if (rs > 0) v = rs > 54 ? 0 : shift_even(m, rs);
  if (eb == 0) v = 0;
  return x < 0.0 ? -v : v;
}

// x 2^(62-e) as an integer (|x| < 2^e): every bit of entries down to 2^-9 of
// the row's power of two, rounded to nearest below.
__device__ __forceinline__ long long sfixed62(double x, int e) {
  const uint64_t bits = (uint64_t)__double_as_longlong(x);
  const int eb = (int)((bits >> 52) & 0x7ff);
  const uint64_t m = (bits & ((1ULL << 52) - 1)) | (1ULL << 52);
  const int rs = e - (eb - 1022) - 9;  // |x| 2^(62-e) = m 2^-rs
  long long v = (long long)(m << min(max(-rs, 0), 9));
  if (rs > 0) v = rs > 54 ? 0 : (long long)((m + (1ULL << (rs - 1))) >> rs);
  if (eb == 0) v = 0;
  return x < 0.0 ? -v : v;
}

// Largest exponents of rows g and g + 8 of a warp's (half) tile, gathered per
// column half: ex[row].
__device__ __forceinline__ void put_row_exps(int* ex, int ti, int lane, int e0, int e1) {
#pragma unroll
  for (int off = 1; off <= 2; off <<= 1) {
    e0 = max(e0, __shfl_xor_sync(0xffffffffu, e0, off));
    e1 = max(e1, __shfl_xor_sync(0xffffffffu, e1, off));
  }
  if ((lane & 3) == 0) {
    ex[ti * 16 + (lane >> 2)] = e0;
    ex[ti * 16 + (lane >> 2) + 8] = e1;
  }
}
// The row's exponent over the N warps that share it; ex is [N][mp].
template <int N>
__device__ __forceinline__ int row_exp(const int* ex, int mp, int row) {
  int e = ex[row];
#pragma unroll
  for (int k = 1; k < N; ++k) e = max(e, ex[k * mp + row]);
  return e;
}

// Two digits (fields of 9 bits, 10 at the top) as FP16 halves: (1024 + f) -
// 1280 = f - 256, exact.
__device__ __forceinline__ uint32_t field_pair(uint32_t f0, uint32_t f1) {
  const uint32_t biased = (0x6400u | f0) | ((0x6400u | f1) << 16);
  __half2 h;
  memcpy(&h, &biased, 4);
  h = __hsub2(h, __floats2half2_rn(1280.0f, 1280.0f));
  uint32_t r;
  memcpy(&r, &h, 4);
  return r;
}

// A lane's words of one plane to their place (s: odd octet).
template <int NE>
__device__ __forceinline__ void put_words(const uint32_t* w, uint4* d, int s, int half) {
  if (NE == 8) {
    *d = s ? make_uint4(w[1], w[3], w[0], w[2]) : make_uint4(w[0], w[2], w[1], w[3]);
  } else {
    uint32_t* d32 = reinterpret_cast<uint32_t*>(d);
    d32[2 * s + half] = w[0];
    d32[2 * (1 - s) + half] = w[1];
  }
}

// Writes the top n digits of a lane's 2 NE values (NE real parts, then NE
// imaginary parts; NE = 8: the whole tile, NE = 4: its column half `half`) to
// the planes: real parts in planes 0..n-1, imaginary parts in planes
// np..np+n-1, `plane` uint4 apart.  The values are signed fixed point of BITS
// bits after a right shift by sh (a left shift when negative).  The words of
// a digit that gets no plane (n = D - 1) go to `last`, when given.
// With NP = 2 the lane has only the NE values of part `part0` (0 re, 1 im).
template <int BITS, int NE, int NP = 1>
__device__ __forceinline__ void put_planes(const long long* x, int n, uint4* dst, int plane, int np, int half,
                                           int sh = 0, uint32_t* last = nullptr, int part0 = 0) {
  constexpr int D = (BITS - 8) / kDigitBits + 1;  // digits of the format
  const int s = (threadIdx.x >> 3) & 1;           // odd octet: pairs swapped
  long long bias = 0;
#pragma unroll
  for (int p = 0; p < D; ++p) bias += 256LL << (kDigitBits * p);
#pragma unroll
  for (int part = 0; part < 2 / NP; ++part) {
    unsigned long long y[NE];
#pragma unroll
    for (int k = 0; k < NE; ++k) {
      const long long v = x[NE * part + k];
      y[k] = (unsigned long long)((sh >= 0 ? v >> min(sh, 63) : v << min(-sh, 63)) + bias);
    }
#pragma unroll
    for (int p = 0; p < D; ++p) {
      if (p < n || last) {
        uint32_t w[NE / 2];  // words (rows g, g + 8) of each column half
#pragma unroll
        for (int k = 0; k < NE / 2; ++k) {
          const uint32_t mask = p ? 511u : 1023u;
          w[k] = field_pair((uint32_t)(y[2 * k] >> (kDigitBits * (D - 1 - p))) & mask,
                            (uint32_t)(y[2 * k + 1] >> (kDigitBits * (D - 1 - p))) & mask);
        }
        if (p < n) {
          put_words<NE>(w, dst + ((NP == 2 ? part0 : part) * np + p) * plane, s, half);
        } else {
#pragma unroll
          for (int k = 0; k < NE / 2; ++k) last[part * (NE / 2) + k] = w[k];
        }
      }
    }
  }
}

// hi 2^sh + lo 2^(sh - 36), truncated, as an integer (it must fit).
__device__ __forceinline__ long long fix_shift(long long hi, long long lo, int sh) {
  hi += lo >> 36;
  const unsigned long long f = ((unsigned long long)lo << 28) >> 1;  // fraction below hi, 63 bits
  const int s = min(max(sh, 0), 63);
  const long long r = (hi << s) | (long long)(f >> (63 - s));
  return r >> min(max(-sh, 0), 63);
}

// x 2^e rounded to nearest (ties to even), in integer instructions: FP64
// conversions and scalings cost an FP64 issue slot each.  Zero below the
// normal range.
__device__ __forceinline__ double fix_to_double(long long x, int e) {
  const unsigned long long m = (unsigned long long)(x < 0 ? -x : x);
  const int lz = __clzll((long long)m);
  const unsigned long long n = m << (lz & 63);  // top bit at 63
  const unsigned rest = (unsigned)n & 0x7ffu, odd = (unsigned)(n >> 11) & 1u;
  const unsigned long long mant = (n >> 11) + ((rest + odd + 0x3ffu) >> 11);
  const int be = e + 63 - lz + 1023;
  if (m == 0 || be < 1) return 0.0;
  if (be > 2046) return __longlong_as_double((long long)((x < 0 ? 1ULL << 63 : 0ULL) | 0x7ff0000000000000ULL));
  return __longlong_as_double((long long)((x < 0 ? 1ULL << 63 : 0ULL) + ((unsigned long long)(be - 1) << 52) + mant));
}

// 2^e (hi 2^-34 + lo 2^-70), rounded once from 62 significant bits.
__device__ __forceinline__ double fold_to_double(long long hi, long long lo, int e) {
  hi += lo >> 36;
  const unsigned long long f = ((unsigned long long)lo << 28) >> 1;
  const int s = min(36, __clzll(hi < 0 ? ~hi : hi) - 2);  // |hi| 2^s < 2^62
  return fix_to_double((hi << s) | (long long)(f >> (63 - s)), e - 34 - s);
}

// The sums hi, lo of one 16 x 8 half of a tile of A B^T' (B in transposed
// planes, see above): levels 0..LMAX of NA and NB digits.  a0 and a1 point at
// the lane's word pairs (a0, a2) and (a1, a3) of the tile row's first tile, b
// at the pair of the wanted half of the tile column's first tile; SA, SB are
// the bytes between real and imaginary planes, `plane` those of a plane.
// Element w of re (im) is hi[w] (hi[4 + w]), in the accumulator layout.
// Three levels are summed side by side, so an A digit serves three B digits
// and each B digit is loaded once per group: 128 bytes of shared memory per
// mma.sync, half of what one level at a time reads (which is the rate at
// which shared memory, not the tensor pipe, is the limit).  A level of n
// digit pairs adds at most n 2^21 per k tile: with up to four pairs a level
// the sums of two k tiles stay within 2^24, and are folded together.
// A seventh digit of B (NB = 7) has its real plane at b6 and its imaginary
// plane after it.
template <int T, int NA, int NB, int LMAX, int NP = 1>
__device__ __forceinline__ void half_product(const char* a0, const char* a1, int SA, const char* b, int SB, int plane,
                                             long long* hi, long long* lo, const char* b6 = nullptr, int part = 0) {
  constexpr int NV = 8 / NP;  // sums of a lane
  // NP = 2, by part: A_re meets B_re or B_im, A_im meets -B_im or B_re
  const uint32_t neg = NP == 2 && part ? 0u : 0x80008000u;
#pragma unroll
  for (int k = 0; k < NV; ++k) hi[k] = lo[k] = 0;
#pragma unroll
  for (int L = 0; L <= LMAX; L += 3) {
    const int top = L + 2 < LMAX ? L + 2 : LMAX;
    // most digit pairs of a level of the group
    int np = 0;
#pragma unroll
    for (int l = L; l <= top; ++l) {
      int c = 0;
#pragma unroll
      for (int p = 0; p < NA; ++p) c += (l - p >= 0 && l - p < NB) ? 1 : 0;
      np = c > np ? c : np;
    }
    const int KF = np <= 4 && T > 1 ? 2 : 1;  // k tiles per fold
#pragma unroll 1
    for (int tk0 = 0; tk0 < T; tk0 += KF) {
      float acc[3][NV];
#pragma unroll
      for (int v = 0; v < 3; ++v)
#pragma unroll
        for (int w = 0; w < NV; ++w) acc[v][w] = 0.0f;
#pragma unroll 1
      for (int tk = tk0; tk < tk0 + KF && tk < T; ++tk) {
        const char* pa0 = a0 + tk * 512;
        const char* pa1 = a1 + tk * 512;
        const char* pb = b + tk * 512;
        uint2 br[3], bi[3];
#pragma unroll
        for (int q = 0; q < NB; ++q)  // the digits the first A digit meets
          if (q >= L && q <= top) {
            const char* pq = q == 6 ? b6 + tk * 512 : pb + q * plane;
            const int im = q == 6 ? plane : SB;
            br[q % 3] = *reinterpret_cast<const uint2*>(pq + (NP == 2 && part ? im : 0));
            bi[q % 3] = *reinterpret_cast<const uint2*>(pq + (NP == 2 && part ? 0 : im));
          }
#pragma unroll
        for (int p = 0; p < NA; ++p) {
          if (p > 0 && L - p >= 0 && L - p < NB) {
            br[(L - p) % 3] = *reinterpret_cast<const uint2*>(pb + (NP == 2 && part ? SB : 0) + (L - p) * plane);
            bi[(L - p) % 3] = *reinterpret_cast<const uint2*>(pb + (NP == 2 && part ? 0 : SB) + (L - p) * plane);
          }
          if (top - p >= 0 && L - p < NB) {
            const uint2 r0 = *reinterpret_cast<const uint2*>(pa0 + p * plane);
            const uint2 r1 = *reinterpret_cast<const uint2*>(pa1 + p * plane);
            const uint2 i0 = *reinterpret_cast<const uint2*>(pa0 + SA + p * plane);
            const uint2 i1 = *reinterpret_cast<const uint2*>(pa1 + SA + p * plane);
            const uint4 ar = make_uint4(r0.x, r1.x, r0.y, r1.y), ai = make_uint4(i0.x, i1.x, i0.y, i1.y);
#pragma unroll
            for (int v = 0; v < 3; ++v) {
              const int q = L + v - p;
              if (q >= 0 && q < NB && L + v <= LMAX) {
                mma16816(acc[v], ar, br[q % 3].x, br[q % 3].y);
                if (NP == 1) mma16816(acc[v] + 4 % NV, ar, bi[q % 3].x, bi[q % 3].y);
              }
            }
#pragma unroll
            for (int v = 0; v < 3; ++v) {
              const int q = L + v - p;
              if (q >= 0 && q < NB && L + v <= LMAX) {
                mma16816(acc[v], ai, bi[q % 3].x ^ neg, bi[q % 3].y ^ neg);
                if (NP == 1) mma16816(acc[v] + 4 % NV, ai, br[q % 3].x, br[q % 3].y);
              }
            }
          }
        }
      }
#pragma unroll
      for (int v = 0; v < 3; ++v)
        if (L + v <= LMAX) {
#pragma unroll
          for (int w = 0; w < NV; ++w) {
            const int x = __float2int_rn(acc[v][w]);
            if (L + v < kHiLevels) hi[w] += (long long)x * (1LL << (kDigitBits * (kHiLevels - 1 - L - v)));
            else lo[w] += (long long)x * (1LL << (kDigitBits * (kLmax - L - v)));
          }
        }
    }
  }
}

}  // namespace oz
}  // namespace rg
