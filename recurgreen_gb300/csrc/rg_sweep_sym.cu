// Symmetric recursive Green sweep for guides of up to 64 modes.
//
// With Dirichlet modes the slice matrix X_n = A_n - V_n - B Gss B is complex
// symmetric (A and B diagonal, V real symmetric, and Gss = inv(X_{n-1}) is
// symmetric in turn).  The kernel keeps it in the variables scaled by
// D = (B/c)^(1/2) (src/waveguide.f90:426-440 in them):
//   X' = D^-1 X D^-1 = c A/B - D^-1 V D^-1 - c G' c,   G' = D Gss D = inv(X'),
//   Q  = (D Gs1 D)^T:  Q_0 = G'_0,  Q_n = -Q_{n-1} c G'_n,
// with c = 1 for open modes, so that a slice needs no product with B, and every
// matrix entry is of order 1.  A closed mode's |A/B| is 2 cosh(kappa dx): on
// coarse slices, where that passes 32, c is the power of two that takes it back
// (the 26 bits of the FP32 inverse do not span cosh(6), and whole items went to
// the pivoted kernel: 304 guides of 63 modes, 14 of them closed, 200 slices,
// kappa dx up to 6.4, 355 ms; 67 now).
//
// In the modes exp(2 pi i k y) of a periodic guide X is Hermitian but for its
// diagonal, not symmetric; A and B depend on |k| alone, so in the real modes
// cos and sin of 2 pi |k| y, a unitary change within each pair k, -k, the same
// recursion is symmetric with the same A and B.  Only V's elements, and t or r
// at the end, differ.  200 guides of 51 modes and 100 slices, t and r: 161 ms
// in the pivoted kernel, 58 to 62 here.
// Periodic items whose states are kept go to the pivoted kernel.
//
// Why not FP64 elimination: FP64 is 1.7 FMA lanes per clock and SM here, so
// the 12 M^3 flops of a Gauss-Jordan sweep on [X | B Gs1] cost 49,000 warp
// instructions of 18 clocks per slice at M = 64 (0.9 M clocks), whatever the
// occupancy.  Instead, per slice:
//   1. to 3. G' = X'^-1 from an FP32 inverse and its residual, exact to
//      FP64, on the FP16 tensor cores (rg_tile_inverse.cuh);
//   4. Q on the tensor cores, all 26 digit pairs, rounded once.
// FP64 instructions are left in the potential's draw and projection, which
// two producer warps run one slice ahead of the others, and in the assembly
// of X'.  The residual makes the result as accurate as an FP64 inverse: against an
// extended-precision sweep the error of t is 0.65 to 1.06 times the elimination's
// (7 to 64 modes, 40 to 300 slices; geometric mean 0.9), that of T 0.4 to 0.95.
// Measured, with the eigenvalues: 304 guides of 64 modes and 600 slices 607 ms
// before, 185 now; 500 of 37 modes and 150 slices 110 ms before, 45 now; one
// guide of 10 modes and 200 slices 8.2 ms before, 2.0 now.
//
// Layout: T = ceil(M/16) tiles a side, one warp per tile or two, as in
// rg_tile_inverse.cuh.  (Q is kept transposed so that it is only ever an A
// operand.)  Its plane regions are reused through the slice:
//   region A: X' -> R -> G';   region B: Y0 -> E_k -> Q.
// Q, G' and the scaling products w_i w_j stay with their owner lanes, in the
// CTA's workspace (L2).  Above 32 modes the registers of one CTA fill an SM (at 48
// modes a warp per tile and two CTAs of 80 registers took the same time).
//
// If a pivot is too small against the unswept entries of its row (sym_tau),
// the residual is not small, or something does not fit its row's fixed point
// (strong disorder), the item is flagged (kStatusNeedPivot), its
// index appended to a.flag_list, and it is recomputed by the pivoted kernel,
// which launch_sweep starts on that list.
#include "rg_tile_inverse.cuh"

namespace rg {
namespace {

__device__ __forceinline__ void bar_sync(int id, int n) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int n) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// Named barriers: the main warps, the producer warps, the two buffers of
// projection coefficients (filled / free again), the propagator's warps, and
// the two buffers of G' for them.
constexpr int kBarMain = 1, kBarProd = 2, kBarFull = 3, kBarFree = 5, kBarProp = 7, kBarGFull = 8, kBarGFree = 10;

// Element (i, j) of modal^T diag(U) modal in the real modes of the guide from
// its projection coefficients co.  Dirichlet: co[d] = cos coefficient d.
// Periodic: co[2 d] and co[2 d + 1] are the cos and sin coefficients of d; mode
// i stands for k = i - M/2: sqrt(2) cos(2 pi k y) for k > 0, sqrt(2)
// sin(2 pi |k| y) for k < 0, and 1.
__device__ __forceinline__ double potential_element(const double* co, int i, int j, int M, bool per) {
  if (!per) return co[i > j ? i - j : j - i] - co[i + j + 2];
  const int ki = i - (M >> 1), kj = j - (M >> 1);
  const int p = ki < 0 ? -ki : ki, q = kj < 0 ? -kj : kj;
  const int odd = (ki < 0) != (kj < 0);
  const double diff = co[2 * (p > q ? p - q : q - p) + odd], sum = co[2 * (p + q) + odd];
  double v;
  if (odd) v = (ki < 0 ? p >= q : q >= p) ? sum + diff : sum - diff;  // the sin index against the cos index
  else v = ki < 0 ? diff - sum : diff + sum;
  if (ki == 0 || kj == 0) v *= ki == kj ? 0.5 : 0.70710678118654752440;
  return v;
}

// Element (i, j) of a matrix in the modes exp(2 pi i k y) of a periodic guide
// from F, the matrix in its real modes (see potential_element).
__device__ __forceinline__ double2 from_real_modes(const double2* F, int ld, int M, int i, int j) {
  const int K = M >> 1, ki = i - K, kj = j - K;
  const int ci = ki < 0 ? K - ki : i, cj = kj < 0 ? K - kj : j;  // the cos modes; the sin modes lie at 2 K - ci
  auto row = [&](int col) {
    const double2 c = F[ci * ld + col];
    if (ki == 0) return c;
    const double2 s = F[(2 * K - ci) * ld + col];
    const double f = ki > 0 ? 1.0 : -1.0;  // (c - i f s) / sqrt(2)
    return cscale(0.70710678118654752440, make_double2(c.x + f * s.y, c.y - f * s.x));
  };
  const double2 c = row(cj);
  if (kj == 0) return c;
  const double2 s = row(2 * K - cj);
  const double f = kj > 0 ? 1.0 : -1.0;  // (c + i f s) / sqrt(2)
  return cscale(0.70710678118654752440, make_double2(c.x - f * s.y, c.y + f * s.x));
}

// PROP: Q has warps of its own, as many as hold the matrix, one slice behind
// the main ones.  Q_n does not feed the recursion of G', so a slice's chain is
// then the inverse alone.  They cost registers and shared memory: at 17 to 32
// modes an SM takes one such CTA instead of two (prop_warps).
template <int T, bool PROP>
struct SymCfg {
  static constexpr int MP = 16 * T;                // padded modes
  static constexpr int NE = T == 4 ? 8 : 4;        // complex entries per lane: a whole tile, or its column half
  static constexpr int NHALF = 8 / NE;             // warps per tile
  // 2: a main warp has one part, re or im, of its entries.  Up to 16 modes, where
  // the instructions of two warps made a slice's latency: one guide of 10 modes
  // and 200 slices 4.85 ms, 3.43 with PROP, 2.07 with both; 600 guides 5.7 ms in
  // any of the forms.
  static constexpr int NP = T == 1 && PROP ? 2 : 1;
  static constexpr int NCW = T * NHALF;            // warps that share a row (main: NP times as many)
  static constexpr int NPROP = 32 * T * T * NHALF;  // threads that hold Q; without PROP the main ones
  static constexpr int NMAIN = NP * NPROP;
  // Producer threads.  Registers are handed out to four warps at a time.
  static constexpr int PROD = T == 4 ? 128 : 64;
  static constexpr int NT = NMAIN + PROD + (PROP ? NPROP : 0);
  static constexpr int MINB = T == 1 || (T == 2 && !PROP) ? 2 : 1;  // CTAs per SM
  static constexpr int PL = T * T * 32;            // uint4 of one digit plane
  static constexpr int LDW = MP + 1;
  static constexpr size_t bytes() {
    return sizeof(uint4) * 24 * PL + sizeof(double) * (2 * (2 * MP + 2) + PROD) + sizeof(unsigned long long) * 2 +
           sizeof(unsigned) * 32 + sizeof(int) * (2 * NP + 1) * NCW * MP +
           (PROP ? sizeof(uint4) * 24 * PL + sizeof(double2) * 2 * NPROP * NE + sizeof(int) * 2 * MP : 0);
  }
};

// Workspace of one CTA in double2: generator states (ny x 4 uint64), the
// potential row, then Q, G' and w_i w_j by warp, element and lane.
inline int64_t sym_stride(int T, int max_ny) {
  return (2 * (int64_t)max_ny + (max_ny + 1) / 2 + 3 * (int64_t)T * T * 256 + 15) & ~(int64_t)15;
}

template <int T, bool PROP>
__global__ void __launch_bounds__(SymCfg<T, PROP>::NT, SymCfg<T, PROP>::MINB) sweep_sym_kernel(SweepArgs a) {
  using Cf = SymCfg<T, PROP>;
  constexpr int MP = Cf::MP, NMAIN = Cf::NMAIN, NT = Cf::NT, PL = Cf::PL, LDW = Cf::LDW, kProd = Cf::PROD;
  constexpr int NE = Cf::NE, NHALF = Cf::NHALF, NCW = Cf::NCW, NP = Cf::NP, NPROP = Cf::NPROP, NV = 2 * NE / NP;
  extern __shared__ uint4 smem[];
  uint4* regA = smem;                          // 12 planes
  uint4* regB = smem + 12 * PL;                // 12 planes
  double* cc = (double*)(smem + 24 * PL);      // [2][2 MP + 2] projection coefficients
  double* psum = cc + 2 * (2 * MP + 2);        // [kProd] partial projections
  unsigned long long* rsum = (unsigned long long*)(psum + kProd);  // [2] sum of squares of the residual
  unsigned* red = (unsigned*)(rsum + 2);       // [32] maxima of a slice
  int* exX = (int*)(red + 32);                 // [NCW][MP] row exponents by warp column: X',
  int* exY = exX + NP * NCW * MP;              // Y0,
  int* exQ = exY + NP * NCW * MP;              // Q
  // of the propagator's warps: [24] planes (G', Q), [2][NPROP NE] G', [2][MP] its row exponents
  uint4* regC = (uint4*)(((size_t)(exQ + NCW * MP) + 15) & ~(size_t)15);
  double2* gbuf = (double2*)(regC + 24 * PL);
  int* eybuf = (int*)(gbuf + 2 * NPROP * NE);
  __shared__ int s_r;
  __shared__ volatile int s_status, s_abort[2], s_gabort[2];
  __shared__ WgDesc wd;

  const int tid = threadIdx.x, lane = tid & 31;
  const bool main_thread = tid < NMAIN, prop_thread = PROP && tid >= NMAIN + kProd;
  const bool out_thread = PROP ? prop_thread : main_thread;  // has whole elements of the results
  const int part = NP == 2 && main_thread ? (tid >> 5) & 1 : 0;
  const int warp = prop_thread ? (tid - NMAIN - kProd) >> 5 : (tid >> 5) / NP;
  const int g = lane >> 2, t4 = lane & 3;
  const int tile = warp / NHALF, half = NHALF == 2 ? warp & 1 : 0;
  const int ti = tile / T, tj = tile % T;
  const int r0 = ti * 16 + g, c0 = tj * 16 + 2 * t4 + 8 * half;
  double2* ws = a.work + (int64_t)blockIdx.x * a.work_stride;
  uint64_t* gen = (uint64_t*)ws;               // [max_ny][4]
  double* urow = (double*)(ws + 2 * (int64_t)a.max_ny);  // [max_ny] potential row
  double2* Qs = ws + 2 * (int64_t)a.max_ny + (a.max_ny + 1) / 2;
  if (main_thread || prop_thread) Qs += warp * 32 * NE + lane;
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

  const TileSmem ts{regA, regB, red, rsum, exX, exY};
  auto mbar = [&]() { bar_sync(kBarMain, NMAIN); };

  for (;;) {
    if (tid == 0) {
      s_r = atomicAdd(a.work_counter, 1);
      if (s_r < a.nreal) wd = a.wgs[a.item_wg ? a.item_wg[s_r] : 0];
    }
    __syncthreads();
    const int r = s_r;
    if (r >= a.nreal) break;
    const int M = wd.M, ny = wd.ny, nx = wd.nx;
    const bool per = wd.periodic != 0;
    const bool pass_on = per && a.state_dump;
    const bool scaled = wd.csc != nullptr;
    if (tid == 0) {
      s_status = pass_on ? kStatusNeedPivot : RG_OK;
      s_abort[0] = s_abort[1] = 0;
    }
    __syncthreads();

    if (pass_on) {
      // handed to the pivoted kernel below
    } else if (prop_thread) {
      // Q, one slice behind the main warps, in this lane's registers.
      double2 q[NE];
      const char* bC = (const char*)regC;
      const char* bD = (const char*)(regC + 12 * PL);
      auto pbar = [&]() { bar_sync(kBarProp, NPROP); };
      for (int n = 0; n < nx && !refl; ++n) {
        const int b = n & 1;
        bar_sync(kBarGFull + b, NMAIN + NPROP);
        const bool skip = s_gabort[b] != 0;
        double2 gd[NE];
        int ec[NE];  // by column of an element
        const int ey0 = eybuf[b * MP + r0], ey1 = eybuf[b * MP + r0 + 8];
#pragma unroll
        for (int k = 0; k < NE; ++k) {
          gd[k] = gbuf[(b * (NPROP / 32) + warp) * 32 * NE + 32 * k + lane];
          ec[k] = eybuf[b * MP + c0 + ecol(k)];
        }
        if (n <= nx - 3) bar_arrive(kBarGFree + b, NMAIN + NPROP);
        if (skip) continue;
        if (n > a.inject_at) {
          if (scaled) {  // Q c (the factors of the padding are 1)
#pragma unroll
            for (int k = 0; k < NE; ++k) q[k] = cscale(wd.csc[c0 + ecol(k)], q[k]);
          }
          int eq0 = oz::kNoExp, eq1 = oz::kNoExp;
#pragma unroll
          for (int k = 0; k < NE; ++k) {
            if (erow(k)) eq1 = max(eq1, oz::fexp2(q[k]));
            else eq0 = max(eq0, oz::fexp2(q[k]));
          }
          pbar();  // the last slice's planes and exponents have been read
          oz::put_row_exps(exQ + (tj * NHALF + half) * MP, ti, lane, eq0, eq1);
          long long acc[2 * NE];
#pragma unroll
          for (int k = 0; k < NE; ++k) {
            acc[k] = oz::sfixed53(gd[k].x, erow(k) ? ey1 : ey0);
            acc[NE + k] = oz::sfixed53(gd[k].y, erow(k) ? ey1 : ey0);
          }
          oz::put_planes<53, NE>(acc, 6, regC + own, PL, 6, half);
          pbar();
          eq0 = oz::row_exp<NCW>(exQ, MP, r0);
          eq1 = oz::row_exp<NCW>(exQ, MP, r0 + 8);
#pragma unroll
          for (int k = 0; k < NE; ++k) {
            const int e = erow(k) ? eq1 : eq0;
            acc[k] = oz::sfixed53(q[k].x, e);
            acc[NE + k] = oz::sfixed53(q[k].y, e);
          }
          oz::put_planes<53, NE>(acc, 6, regC + 12 * PL + own, PL, 6, half);
          pbar();
#pragma unroll
          for (int h = 0; h < NE / 4; ++h) {
            long long hi[8], lo[8];
            oz::half_product<T, 6, 6, oz::kLmax>(bD + offA0, bD + offA1, 6 * kPlane, bC + offB + 8 * (odd ^ (half | h)),
                                                 6 * kPlane, kPlane, hi, lo);
#pragma unroll
            for (int w = 0; w < 4; ++w) {
              const int k = 4 * h + w, e = (erow(k) ? eq1 : eq0) + ec[k];
              q[k] = make_double2(-oz::fold_to_double(hi[w], lo[w], e), -oz::fold_to_double(hi[4 + w], lo[4 + w], e));
            }
          }
        } else {
          // the source slice: Q = G'; zero before it
#pragma unroll
          for (int k = 0; k < NE; ++k) q[k] = n == a.inject_at ? gd[k] : make_double2(0.0, 0.0);
        }
        if (a.state_dump) {
          // as below: Gss = w G' w and Gs1 = w Q^T w
          double2* d1 = a.state_dump + ((int64_t)r * nx + n) * 2 * M * M;
#pragma unroll
          for (int k = 0; k < NE; ++k) {
            const int i = r0 + erow(k), j = c0 + ecol(k);
            if (i < M && j < M) {
              const double2 w = cmul(wd.wsc[i], wd.wsc[j]);
              d1[(int64_t)i * M + j] = cmul(w, gd[k]);
              d1[(int64_t)M * M + (int64_t)j * M + i] = cmul(w, q[k]);
            }
          }
        }
      }
      if (!refl) {
#pragma unroll
        for (int k = 0; k < NE; ++k) Qs[32 * k] = q[k];
      }
    } else if (!main_thread) {
      // Producers: the potential row of slice n and its projection
      // cc[d] = sum_j tab[j][d] U_j, one slice ahead.  The transverse grid
      // is symmetric (y_{ny-1-j} = 1 - y_j) and cos(pi d (1 - y)) =
      // (-1)^d cos(pi d y), so the points pair up as sums (even d) and
      // differences (odd d) over half the points.  (Of a periodic guide the
      // even columns are cos(2 pi d/2 y), the odd ones sin: the same pairs.)
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
      const int h = ny >> 1, nd = per ? 2 * M : 2 * M + 1;
      const double* tab = per ? (const double*)wd.expfac : wd.costab;  // [ny][nd]
      for (int n = 0; n < nx; ++n) {
        const int b = n & 1;
        if (n >= 2) bar_sync(kBarFree + b, NMAIN + kProd);
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
            const double* ct = tab + d;
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
            if (seg < nseg) psum[pt] = dot(d, seg * h / nseg, (seg + 1) * h / nseg, seg == nseg - 1);
            bar_sync(kBarProd, kProd);
            if (pt < nd) {
              double s = psum[pt];
              for (int k = 1; k < nseg; ++k) s += psum[k * nd + pt];
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
              const double* ct = tab + d;
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
        bar_arrive(kBarFull + b, NMAIN + kProd);
      }
    } else {
      // Scaling products w_i w_j of this lane's elements.
      bool real_w = true;
#pragma unroll
      for (int k = 0; k < NE; ++k) {
        const int i = r0 + erow(k), j = c0 + ecol(k);
        double2 v = make_double2(0.0, 0.0);
        if (i < M && j < M) v = cmul(wd.wsc[i], wd.wsc[j]);
        if (part == 0) Ww[32 * k] = v;
        real_w = real_w && v.y == 0.0;
      }
      real_w = __all_sync(0xffffffffu, real_w);
      double* gp = reinterpret_cast<double*>(Gs) + part;  // value q of this lane: part of element q mod NE
      const double* wp = reinterpret_cast<const double*>(Ww) + part;
      mbar();  // Ww is complete
      bool aborted = false;
      for (int n = 0; n < nx; ++n) {
        const int b = n & 1;
        bar_sync(kBarFull + b, NMAIN + kProd);
        double x[NV];
        if (!aborted) {
          if (scaled && n > 0) {  // c G' c and Q c in place (the factors of the padding are 1)
#pragma unroll 1
            for (int k = 0; k < NE; ++k) {
              const double cj = wd.csc[c0 + ecol(k)], f = wd.csc[r0 + erow(k)] * cj;
              gp[64 * k] *= f;
              if (NP == 1) gp[64 * k + 1] *= f;
              if (!PROP && !refl) Qs[32 * k] = cscale(cj, Qs[32 * k]);
            }
          }
          // 1. X' = c A/B - w V w - c G' c (zero outside M x M).
          const int id = (refl ? nx - 1 - n : n) - wd.nxfree;
          const bool dis = (id >= 0 && id < wd.nxdiso), edge = (n == 0 || n == nx - 1);
          const double* co = cc + b * (2 * MP + 2);
          const double* aw = (const double*)(edge ? wd.aw_edge : wd.aw_bulk);
#pragma unroll
          for (int k = 0; k < NE; ++k) {
            const int i = r0 + erow(k), j = c0 + ecol(k);
            const bool on = i < M && j < M;
            const double vij = on && dis ? potential_element(co, i, j, M, per) : 0.0;
#pragma unroll
            for (int q = k; q < NV; q += NE) {
              const int p = q < NE ? part : 1;  // this value's part
              double v = 0.0;
              if (on) {
                if (n > 0) v = -gp[64 * k + (q < NE ? 0 : 1)];
                if (i == j) v += aw[2 * i + p];
                if (dis && (p == 0 || !real_w)) v = fma(-wp[64 * k + (q < NE ? 0 : 1)], vij, v);
                if (i == j) v += aw[2 * (M + i) + p];  // the rest of c A/B beyond FP64
              }
              x[q] = v;
            }
          }
        }
        if (n <= nx - 3) {
          if (tid == 0) s_abort[b] = aborted ? 1 : 0;
          bar_arrive(kBarFree + b, NMAIN + kProd);
        }
        const bool hand_on = PROP && !refl;
        if (aborted) {
          if (hand_on) {
            if (n >= 2) bar_sync(kBarGFree + b, NMAIN + NPROP);
            if (tid == 0) s_gabort[b] = 1;
            bar_arrive(kBarGFull + b, NMAIN + NPROP);
          }
          continue;
        }

        // 2. G' = X'^-1 (rg_tile_inverse.cuh).
        const bool prod = !PROP && !refl && n > a.inject_at;
        double2 q[NE];
        double gd[NV];
        int ey0, ey1;
        auto q_exps = [&]() {  // Q, and its row exponents for the others
          if (!prod) return;
          int eq0 = oz::kNoExp, eq1 = oz::kNoExp;
#pragma unroll
          for (int k = 0; k < NE; ++k) {
            q[k] = Qs[32 * k];
            if (erow(k)) eq1 = max(eq1, oz::fexp2(q[k]));
            else eq0 = max(eq0, oz::fexp2(q[k]));
          }
          oz::put_row_exps(exQ + (tj * NHALF + half) * MP, ti, lane, eq0, eq1);
        };
        if (!tile_inverse<T, NE, NP>(x, M, tau, ts, &s_status, &s_status, mbar, q_exps, gd, ey0, ey1)) {
          aborted = true;
          if (hand_on) {
            if (n >= 2) bar_sync(kBarGFree + b, NMAIN + NPROP);
            if (tid == 0) s_gabort[b] = 1;
            bar_arrive(kBarGFull + b, NMAIN + NPROP);
          }
          continue;
        }
        if (hand_on) {
          if (n >= 2) bar_sync(kBarGFree + b, NMAIN + NPROP);
#pragma unroll
          for (int k = 0; k < NV; ++k) {
            double2* d = gbuf + (b * (NPROP / 32) + warp) * 32 * NE + 32 * (k % NE) + lane;
            reinterpret_cast<double*>(d)[k < NE ? part : 1] = gd[k];
          }
          if (tj == 0 && half == 0 && part == 0 && t4 == 0) {
            eybuf[b * MP + r0] = ey0;
            eybuf[b * MP + r0 + 8] = ey1;
          }
          if (tid == 0) s_gabort[b] = 0;
          bar_arrive(kBarGFull + b, NMAIN + NPROP);
        }

        // 3. Q <- -Q G' on the tensor cores.
        long long acc[2 * NE];
#pragma unroll
        for (int k = 0; k < NV; ++k) {
          gp[64 * (k % NE) + k / NE] = gd[k];
          if (prod) acc[k] = oz::sfixed53(gd[k], erow(k % NE) ? ey1 : ey0);
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
              Qs[32 * k] =
                  make_double2(-oz::fold_to_double(hi[w], lo[w], e), -oz::fold_to_double(hi[4 + w], lo[4 + w], e));
            }
          }
        } else if (!PROP && !refl) {
          // the source slice: Q = G'; zero before it
#pragma unroll
          for (int k = 0; k < NE; ++k) Qs[32 * k] = n == a.inject_at ? Gs[32 * k] : make_double2(0.0, 0.0);
        }
        if (a.state_dump && !hand_on) {
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
      double2* F = (double2*)regB;  // [MP][LDW] periodic: G11 in the real modes
      if (per) {
        if (out_thread) {
#pragma unroll
          for (int k = 0; k < NE; ++k) F[(r0 + erow(k)) * LDW + c0 + ecol(k)] = cmul(Ww[32 * k], Gs[32 * k]);
        }
        __syncthreads();
      }
      if (out_thread) {
#pragma unroll
        for (int k = 0; k < NE; ++k) {
          const int i = r0 + erow(k), j = c0 + ecol(k);
          if (i < M && j < M) {
            const double2 g11 = per ? from_real_modes(F, LDW, M, i, j) : cmul(Ww[32 * k], Gs[32 * k]);
            const double2 v = cmul(cmul(wd.sqmu_r[i], g11), wd.sqmu_r[j]);
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
    double2* F = (double2*)regB;  // [MP][LDW] periodic: Gs1 in the real modes
    if (per) {
      if (out_thread) {
#pragma unroll
        for (int k = 0; k < NE; ++k) F[(c0 + ecol(k)) * LDW + r0 + erow(k)] = cmul(Ww[32 * k], Qs[32 * k]);
      }
      __syncthreads();
    }
    if (out_thread) {
#pragma unroll
      for (int k = 0; k < NE; ++k) {
        const int gj = r0 + erow(k), gi = c0 + ecol(k);  // Q[j][i]
        const int i = gi - row0, j = gj - col0;
        if (i >= 0 && i < nrow && j >= 0 && j < ncol) {
          const double2 gs1 = per ? from_real_modes(F, LDW, M, gi, gj) : cmul(Ww[32 * k], Qs[32 * k]);
          const double2 v = cmul(cmul(sqmu[gi], gs1), sqmu[gj]);
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

// Whether Q gets warps of its own at 17 to 32 modes: while all realizations run
// at once with them.  32 modes and 150 slices, batches of 1 and 152: 5.1 and 5.2
// ms with, 6.6 without; 200 would need two waves for 7.9 ms.
bool prop_warps(const SweepArgs& a, int sm_count) { return a.nreal <= sm_count; }

template <int T, bool PROP>
int plan_sym_t(SweepArgs& a, int sm_count, int* grid, int64_t* stride) {
  const size_t smem = SymCfg<T, PROP>::bytes();
  const auto kernel = sweep_sym_kernel<T, PROP>;
  RG_CUDA(allow_smem((const void*)kernel, smem));
  int per_sm = 0;
  RG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, SymCfg<T, PROP>::NT, smem));
  if (per_sm < 1) return fail(RG_ERR_INVALID_ARG, "symmetric sweep kernel does not fit on an SM");
  if (a.force_per_sm > 0 && a.force_per_sm < per_sm) per_sm = a.force_per_sm;
  int g = per_sm * sm_count;
  if (g > a.nreal) g = a.nreal;
  *grid = g < 1 ? 1 : g;
  *stride = sym_stride(T, a.max_ny);
  a.cluster = 1;
  a.prop_warps = PROP;
  return RG_OK;
}

template <int T, bool PROP>
int launch_sym_t(const SweepArgs& a, cudaStream_t stream, int grid) {
  sweep_sym_kernel<T, PROP><<<grid, SymCfg<T, PROP>::NT, SymCfg<T, PROP>::bytes(), stream>>>(a);
  RG_CUDA(cudaGetLastError());
  return RG_OK;
}

}  // namespace

int sweep_sym_plan(SweepArgs& a, int sm_count, int* grid, int64_t* work_stride) {
  if (a.max_M <= 16) return plan_sym_t<1, true>(a, sm_count, grid, work_stride);
  if (a.max_M <= 32)
    return prop_warps(a, sm_count) ? plan_sym_t<2, true>(a, sm_count, grid, work_stride)
                                   : plan_sym_t<2, false>(a, sm_count, grid, work_stride);
  if (a.max_M <= 48) return plan_sym_t<3, false>(a, sm_count, grid, work_stride);
  if (a.max_M <= kMaxModesSmem) return plan_sym_t<4, false>(a, sm_count, grid, work_stride);
  return fail(RG_ERR_INVALID_ARG, "symmetric sweep kernel: too many modes");
}

int launch_sweep_sym(const SweepArgs& a, cudaStream_t stream, int grid) {
  if (a.nreal <= 0) return RG_OK;
  if (a.max_M <= 16) return launch_sym_t<1, true>(a, stream, grid);
  if (a.max_M <= 32)
    return a.prop_warps ? launch_sym_t<2, true>(a, stream, grid) : launch_sym_t<2, false>(a, stream, grid);
  if (a.max_M <= 48) return launch_sym_t<3, false>(a, stream, grid);
  return launch_sym_t<4, false>(a, stream, grid);
}

}  // namespace rg
