// bdhi_kernel.cu -- Brownian dynamics with hydrodynamic interactions
// (Ermak-McCammon, i_simulate_type = BROWNIAN_HI), batched over lanes of
// different sizes, FP64 (precision 1: Cholesky trailing updates on the
// tensor cores in split TF32).
//
// One step of time_integral.F90:429-457 for every lane:
//   [every n_step_hydro steps] D = RPY tensor at x (simu_hydro_tensors.F90:
//       139-182, HI_TENSOR%RPY), L = Cholesky factor of D (:304-324):
//       rpy_kernel, chol_diag_kernel (L_00), then per 64-wide panel k:
//       chol_panel_kernel (L_ik = A_ik L_kk^-T below the diagonal tile) and
//       chol_update_kernel or chol_update_tc_kernel (A_ij -= L_ik L_jk^T for
//       the trailing tiles, FP64 or tensor cores; the CTA that finishes tile
//       (k + 1, k + 1) factors it for the next panel)
//   bd_noise_kernel     xi (counter-based or injected r_boxmuller)
//   bd_update_kernel    dx_k = tstep/kT (D F)_k + sqrt(2 tstep) (L xi)_k,
//                       x += dx (one warp per row, HBM-bound matrix-vector)
//   bd_force_kernel     F = FENE + WCA at the new x (force_fene.F90,
//                       force_wca.F90): one warp per bead gathers its records
//
// Matrices are row-major (3N x 3N) per lane at lane.bd0.  Sums run in a fixed
// order (warp butterflies, per-thread loops), so results do not depend on
// scheduling.  A pivot <= 0 sets the lane's not_spd flag (the reference stops
// with util_error); the factorisation continues with a unit pivot so that no
// NaN spreads, and the host reports TIS_E_NOT_SPD.
#include "device_common.cuh"

#include <algorithm>
#include <vector>

namespace tis {

constexpr int CT = 64;          // Cholesky tile
// row of an operand tile in shared memory: 136 words, so the 4 x 4 doubles of
// a half-warp's matrix fragment lie in different banks
constexpr int CTP = CT + 4;
constexpr int BD_SMS = 148;

// ------------------------------------------------------------ RPY tensor
// The 3x3 block pre1 I + pre2 r r^T of the bead pair (i < j, r = x_j - x_i)
// in simu_hydro_tensors.F90:50-300, each variant's expressions in the
// reference's evaluation order with explicitly rounded operations (the FP64
// D is bit-identical to the reference's arithmetic).  diag_only: the block
// is val I (Zuk-RPY, one bead inside the other).
struct HiBlock { double pre1, pre2; bool diag_only; };

__device__ __forceinline__ HiBlock hi_pair(int type, double rad, double rad_i, double rad_j, double r_sq, double c6,
                                           double c8) {
  const double r_abs = sqrt(r_sq);
  HiBlock b{0.0, 0.0, false};
  auto rpy = [&](double rs) {   // rad_sq-sum form shared by RPY and Zuk-RPY apart
    b.pre1 = __dmul_rn(__ddiv_rn(c8, r_abs), __dadd_rn(1.0, __ddiv_rn(rs, __dmul_rn(3.0, r_sq))));
    b.pre2 = __ddiv_rn(__dmul_rn(__ddiv_rn(c8, r_abs), __dsub_rn(1.0, __ddiv_rn(rs, r_sq))), r_sq);
  };
  if (type == TIS_HI_ZUK_RPY_DEV) {
    if (__dadd_rn(rad_i, rad_j) < r_abs) {
      rpy(__dadd_rn(__dmul_rn(rad_i, rad_i), __dmul_rn(rad_j, rad_j)));
    } else {
      const double rad_s = rad_i < rad_j ? rad_i : rad_j, rad_l = rad_i < rad_j ? rad_j : rad_i;
      if (__dsub_rn(rad_l, rad_s) < r_abs) {
        const double r_cb = __dmul_rn(r_sq, r_abs);
        const double dr = __dsub_rn(rad_i, rad_j), dr2 = __dmul_rn(dr, dr);
        const double y1 = __dadd_rn(dr2, __dmul_rn(3.0, r_sq));
        const double x1 = __dsub_rn(__dmul_rn(__dmul_rn(16.0, r_cb), __dadd_rn(rad_i, rad_j)), __dmul_rn(y1, y1));
        const double cij = __ddiv_rn(__ddiv_rn(c6, rad_i), rad_j);
        b.pre1 = __ddiv_rn(__ddiv_rn(__dmul_rn(cij, x1), 32.0), r_cb);
        const double y2 = __dsub_rn(dr2, r_sq);
        b.pre2 = __ddiv_rn(__ddiv_rn(__ddiv_rn(__dmul_rn(__dmul_rn(cij, 3.0), __dmul_rn(y2, y2)), 32.0), r_cb), r_sq);
      } else {
        b.pre1 = __ddiv_rn(c6, rad_l);
        b.diag_only = true;
      }
    }
    return b;
  }
  const double rad_sq = __dmul_rn(rad, rad);
  if (type == TIS_HI_RPY_DEV || __dmul_rn(2.0, rad) < r_abs) {
    rpy(__dmul_rn(2.0, rad_sq));
  } else if (type == TIS_HI_RPY_OVER_DEV) {
    b.pre1 = __dmul_rn(__ddiv_rn(c6, rad), __dsub_rn(1.0, __ddiv_rn(__dmul_rn(0.28125, r_abs), rad)));
    b.pre2 = __ddiv_rn(__ddiv_rn(__ddiv_rn(__dmul_rn(__ddiv_rn(c6, rad), 3.0), 32.0), rad), r_abs);
  } else {   // ERMAK_OVER
    b.pre1 = __ddiv_rn(__dmul_rn(__ddiv_rn(__ddiv_rn(c8, 2.0), rad), 7.0), 6.0);
    b.pre2 = __ddiv_rn(__ddiv_rn(__ddiv_rn(c8, 2.0), 2.0), r_sq);
  }
  return b;
}

// grid (ceil(N*N / 256), nlane): thread per ordered bead pair (i, j); writes
// the 3x3 block of D and the lower part of L (L = tril(D) before factoring)
__global__ void __launch_bounds__(256) rpy_kernel(KArgs a) {
  const int lane = blockIdx.y;
  if (lane >= a.nlane) return;
  const LaneDesc L = a.lanes[lane];
  const TopDesc Tp = a.tops[L.top];
  const int N = Tp.nmp, n = 3 * N;
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (long long)N * N) return;
  const int i = (int)(e / N), j = (int)(e - (long long)i * N);
  const double T = a.lab_T[a.lstate[lane].label];
  const double c6 = a.boltz * T / (6.0 * a.pi * a.viscosity);
  const double c8 = a.boltz * T / (8.0 * a.pi * a.viscosity);
  const double *hr = a.b_hrad + Tp.bead0;
  const double rad = hr[0];   // radius(1) of RPY, RPY_OVER and ERMAK_OVER
  const int type = a.i_hydro_tensor;
  double blk[3][3];
  if (i == j) {
    const double dv = c6 / (type == TIS_HI_ZUK_RPY_DEV ? hr[i] : rad);
    for (int p = 0; p < 3; ++p)
      for (int q = 0; q < 3; ++q) blk[p][q] = (p == q) ? dv : 0.0;
  } else {
    // the reference fills i < j with r = x_j - x_i and mirrors the block;
    // the block is even in r, so both orders give the same numbers
    const int lo = i < j ? i : j, hi = i < j ? j : i;
    const double *x = a.xyz + 3 * (size_t)L.state0;
    double r[3];
    for (int d = 0; d < 3; ++d) r[d] = __dsub_rn(x[3 * hi + d], x[3 * lo + d]);
    const double r_sq = __dadd_rn(__dadd_rn(__dmul_rn(r[0], r[0]), __dmul_rn(r[1], r[1])), __dmul_rn(r[2], r[2]));
    const HiBlock hb = hi_pair(type, rad, hr[lo], hr[hi], r_sq, c6, c8);
    for (int p = 0; p < 3; ++p)
      for (int q = 0; q < 3; ++q) {
        if (hb.diag_only) blk[p][q] = (p == q) ? hb.pre1 : 0.0;
        else if (p == q) blk[p][q] = __dadd_rn(hb.pre1, __dmul_rn(__dmul_rn(hb.pre2, r[p]), r[q]));
        else blk[p][q] = __dmul_rn(__dmul_rn(hb.pre2, r[p]), r[q]);
      }
  }
  // D in FP64 (or FP32, rows padded to 4, for the mixed-precision step),
  // the lower part of L (its upper part is never read)
  double *Lm = a.bd_L + L.bd0;
  for (int p = 0; p < 3; ++p) {
    const size_t row = (size_t)(3 * i + p) * n + 3 * j;
    for (int q = 0; q < 3; ++q) {
      if (a.bd_tc) a.bd_D32[L.bd32 + (size_t)(3 * i + p) * ((n + 3) & ~3) + 3 * j + q] = (float)blk[p][q];
      else a.bd_D[L.bd0 + row + q] = blk[p][q];
      if (a.bd_refine) a.bd_D64[L.bd0 + row + q] = blk[p][q];
      if (3 * j + q <= 3 * i + p) Lm[row + q] = blk[p][q];
    }
  }
}

// ------------------------------------------------------------ Cholesky
__device__ __forceinline__ int lane_tiles(const KArgs &a, const LaneDesc &L, int &n) {
  n = 3 * a.tops[L.top].nmp;
  return (n + CT - 1) / CT;
}

// TF32 split of an FP64 value: hi keeps the top 10 mantissa bits of the
// FP32 rounding (round half up in magnitude), lo = the FP32 rest
__device__ __forceinline__ void tf32_split(double x, float &hi, float &lo) {
  const float xf = (float)x;
  hi = __uint_as_float((__float_as_uint(xf) + 0x1000u) & 0xFFFFE000u);
  lo = xf - hi;
}

// Panel operand planes for the tensor cores: per lane and panel parity
// (two slots: the wide update reads panels k and k + 1), (T + 1) tiles of
// 64 rows x 64 panel columns of TF32 hi parts, then as many of lo parts
// (tile T stays zero: the partner of an odd last row tile).  Inside a tile
// the layout is the K-major, no-swizzle canonical UMMA layout with 8-row
// groups outermost: float offset of (r, c) = (r / 8) 512 + (c / 4) 32 +
// (r % 8) 4 + c % 4, so consecutive row tiles form one operand of 128 rows.
constexpr int PT = CT * CT;   // floats per plane tile
// shared memory of the FP64 tile kernels: two padded tiles
constexpr int U64_SMEM = 2 * CT * CTP * (int)sizeof(double);

// FP64 matrix instruction, c += a b for 8 x 8 x 4: lane l holds a(l / 4, l % 4),
// b(l % 4, l / 4) and c(l / 4, 2 (l % 4) + {0, 1}).  Its rate is that of the
// FP64 FMAs (64 per SM and cycle, measured), but one 64-bit load per operand
// feeds 8 products: with FMAs on 4 x 4 register tiles the tile products were
// bound by shared memory (96 cycles of loads per 64 of FMAs).
__device__ __forceinline__ void mma8(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

// Load diagonal tile td of a lane for factor_diag_tile: the lower part of the
// matrix, identity beyond it, zeros above the diagonal.
__device__ __forceinline__ void load_diag_tile(const double *Lm, int n, int td, int tid, double (&acc)[8][2]) {
  const int w = tid >> 5, r = (tid & 31) >> 2, k2 = 2 * (tid & 3), i = 8 * w + r, i0 = td * CT;
#pragma unroll
  for (int ct = 0; ct < 8; ++ct)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int c = 8 * ct + k2 + q;
      acc[ct][q] = (c <= i && i0 + i < n) ? Lm[(size_t)(i0 + i) * n + i0 + c] : (i == c ? 1.0 : 0.0);
    }
}

// Factor diagonal tile td of a lane and invert its factor with the 256
// threads of the calling group (tid 0..255, 8 warps; sync() is the group's
// barrier).  Warp w holds rows 8 w .. + 7 of the tile in the accumulator
// layout of mma8: acc[ct] = columns 8 ct .. + 7.
//
// This is the serial chain of a refresh: 64 pivots per panel, one after the
// other, the rest of a small problem's chip idle meanwhile.  Right-looking
// Cholesky in the unscaled form A_ic -= A_ij A_cj / p_j (p_j the pivot, L_ij =
// A_ij / sqrt(p_j)), 8 columns per block:
//   every lane of warps 0..2 factors the block's 8 x 8 diagonal block by
//     itself in registers: a pivot costs its reciprocal, a product and an
//     update, with no shuffle and no barrier between two pivots;
//   thread t < 64 then solves row t of the block's columns against it;
//   all warps apply the block's rank-8 update to the columns to the right, in
//     their accumulators.
// The inverse comes with it: the rows of the identity are appended below the
// matrix and take the same steps, which leaves Lu^-T (Lu the unit lower
// factor).  Row r of it is zero before column r, so it takes the places of the
// tile's upper part, and at every block the 64 threads have one row each: a
// row of the matrix below the block or a row of the identity above.
// In one launch of its own, cold (ncu): 36.8 us when one warp factored 16
// columns for all rows, pivots and columns passed by shuffles, and the inverse
// followed in 64 more steps; 11.9 us this way.
//
// The results are written at the end: with the idle warps writing a block's
// while the next is factored, a block took 900 + 1050 cycles (factor, update)
// instead of 800 + 690.
//
// A pivot <= 0 is replaced by 1 (no NaN spreads) and flags the lane.  Stores
// L_tt (zero above the diagonal; FP32 copy for mixed precision) and, when a
// panel follows, U_tt = L_tt^-T into the lane's inverse slot.  vec holds
// FD_VEC doubles (16-byte aligned).
constexpr int FB = 8;           // columns per block
constexpr int FBP = FB + 4;     // row of a block's columns: fragments without bank conflicts
constexpr int FD_X = (CT + FB) * FBP + 2 * FB + 4;   // a block: rows, the block's own lower rows, pivots, 1 / pivots
constexpr int FD_VEC = CT / FB * FD_X + CT * FBP;
static_assert(FD_VEC * (int)sizeof(double) <= U64_SMEM, "the factor's work space reuses the operand tiles");

// 1 / p for 2^-1021 <= p <= 2^1021: the instruction's approximation (20 bits
// or more) and two Newton-Raphson steps y += y (1 - p y), each doubling its
// bits; at most 1 ulp off (the test takes CUDA's own reciprocal for reference).
// Without the division's branch the updates of one pivot fill the wait of the
// next: 821 us for four steps of 150 beads with a refresh each, 856 with
// __drcp_rn.
constexpr double PIVOT_MIN = 0x1p-1021, PIVOT_MAX = 0x1p1021;
__device__ __forceinline__ double pivot_rcp(double p) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(p));
  y = fma(y, fma(-p, y, 1.0), y);
  return fma(y, fma(-p, y, 1.0), y);
}

// Factor the 8 x 8 block at xin + c0 FBP and solve the thread's row v against
// it; d = pivots, ip = their reciprocals.  Returns true if a pivot is outside
// pivot_rcp's range: the values are then of no use without guard, which divides
// and replaces a pivot that is not > 0 by 1, and returns true if there is one
// (its division, compare and selects are on the chain of every pivot).
template <bool guard>
__device__ __forceinline__ bool diag_block(const double *xin, const double *row, int own, double (&v)[FB],
                                           double (&d)[FB], double (&ip)[FB]) {
  double b[FB][FB + 1];
#pragma unroll
  for (int i = 0; i < FB; ++i)
#pragma unroll
    for (int c = 0; c <= i; c += 2) {
      const double2 x = *(const double2 *)&xin[i * FBP + c];
      b[i][c] = x.x;
      b[i][c + 1] = x.y;
    }
#pragma unroll
  for (int q = 0; q < FB; q += 2) {
    const double2 x = *(const double2 *)&row[q];
    v[q] = own < 0 ? x.x : (q == own ? 1.0 : 0.0);
    v[q + 1] = own < 0 ? x.y : (q + 1 == own ? 1.0 : 0.0);
  }
  bool bad = false;
#pragma unroll
  for (int j = 0; j < FB; ++j) {
    double p = b[j][j], r = guard ? 1.0 / p : pivot_rcp(p);
    const bool ok = guard ? p > 0.0 : p >= PIVOT_MIN && p <= PIVOT_MAX;
    bad |= !ok;
    if (guard && !ok) p = r = 1.0;
    d[j] = p;
    ip[j] = r;
    double m[FB];   // column j of the unit factor
#pragma unroll
    for (int i = j + 1; i < FB; ++i) m[i] = b[i][j] * r;
#pragma unroll
    for (int i = j + 1; i < FB; ++i)
#pragma unroll
      for (int c = j + 1; c <= i; ++c) b[i][c] -= m[i] * b[c][j];
#pragma unroll
    for (int i = j + 1; i < FB; ++i) v[i] -= v[j] * m[i];
  }
  return bad;
}

// Columns to the right of block s: acc -= (X / p) X^T.  acc[j] holds column
// tile s + j on entry and s + 1 + j on return (the products move it one place
// down), whose first goes to xin as block s + 1.  A row of the matrix stops at
// its diagonal, a row of the identity goes to the end; beyond, the operands are
// zero (a branch per column tile cost more than its products).  NJ >= 7 - s
// column tiles.
template <int NJ>
__device__ __forceinline__ void diag_trailing(int s, double (&acc)[8][2], const double *X, double *xin, int tid) {
  const int w = tid >> 5, r = (tid & 31) >> 2, k = tid & 3;
  const double *xa = X + (8 * w + r) * FBP + k, *ip = X + (CT + FB) * FBP + FB;
  const double a0 = -xa[0] * ip[k], a1 = -xa[4] * ip[4 + k];
  const int last = w <= s ? 7 : w;
  double b0[NJ], b1[NJ];
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    const int ct = s + 1 + j;
    const double *xb = X + (8 * min(ct, 7) + r) * FBP + k;
    b0[j] = ct <= last ? xb[0] : 0.0;
    b1[j] = ct <= last ? xb[4] : 0.0;
  }
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    acc[j][0] = acc[j + 1][0];
    acc[j][1] = acc[j + 1][1];
    mma8(acc[j], a0, b0[j]);
  }
#pragma unroll
  for (int j = 0; j < NJ; ++j) mma8(acc[j], a1, b1[j]);
  *(double2 *)&xin[(8 * w + r) * FBP + 2 * k] = make_double2(acc[0][0], acc[0][1]);
}

template <typename Sync>
__device__ void factor_diag_tile(const KArgs &a, int lane, double *Lm, int n, int td, double (&acc)[8][2],
                                 double *vec, int tid, Sync sync) {
  const int r0 = td * CT, nb = min(CT, n - r0), np = (n + 3) & ~3;
  float *L32 = a.bd_tc ? a.bd_L32 + a.lanes[lane].bd32 : nullptr;
  double *wout = r0 + CT < n ? a.bd_W + (size_t)lane * CT * CT : nullptr;   // a panel of rows below follows (then nb = CT)
  double *xin = vec + CT / FB * FD_X;
  bool bad = false;
  sync();   // vec is free
  *(double2 *)&xin[(tid >> 2) * FBP + 2 * (tid & 3)] = make_double2(acc[0][0], acc[0][1]);
#pragma unroll 1
  for (int s = 0; s < CT / FB; ++s) {
    sync();   // xin: the block's columns with all earlier blocks applied
    double *X = vec + s * FD_X;
    if (tid < 96) {
      // threads 0 .. 63: row tid below the block, or the identity's row tid
      // (own: one that starts in this block); 64 .. 71: the block's own rows
      const int o = tid - FB * s, own = tid < CT && (unsigned)o < (unsigned)FB ? o : -1;
      const double *row = xin + (tid < CT ? tid : FB * s + (tid & 7)) * FBP;
      double v[FB], d[FB], ip[FB];
      if (diag_block<false>(xin + FB * s * FBP, row, own, v, d, ip)) {   // the same in every thread
        bad |= diag_block<true>(xin + FB * s * FBP, row, own, v, d, ip);
      }
      if (tid < CT + FB) {
#pragma unroll
        for (int q = 0; q < FB; q += 2) *(double2 *)&X[tid * FBP + q] = make_double2(v[q], v[q + 1]);
      } else if (tid == CT + FB) {
#pragma unroll
        for (int q = 0; q < FB; q += 2) {
          *(double2 *)&X[(CT + FB) * FBP + q] = make_double2(d[q], d[q + 1]);
          *(double2 *)&X[(CT + FB) * FBP + FB + q] = make_double2(ip[q], ip[q + 1]);
        }
      }
    }
    sync();
    if (s < 3) diag_trailing<7>(s, acc, X, xin, tid);
    else if (s + 1 < CT / FB) diag_trailing<4>(s, acc, X, xin, tid);
  }
  // L[i][c] and U[i][c] = (L^-1)[c][i]; thread: column c, rows i0 + 4 u.  A
  // block's column is unscaled: L_ic = x / sqrt(p_c)
  const int c = tid & 63, q = c & 7;
  const double *X = vec + (c >> 3) * FD_X;
  const double d = sqrt(X[(CT + FB) * FBP + q]), ri = 1.0 / d;
  const int i0 = tid >> 6, c8 = c & ~7;
  double u[CT / 4];
#pragma unroll
  for (int t = 0; t < CT / 4; ++t) u[t] = X[(i0 + 4 * t) * FBP + q] * ri;   // L below the block, else U
#pragma unroll
  for (int t = 0; t < FB / 4; ++t) {   // the block's own rows of L
    const int o = i0 + 4 * t, i = c8 + o;
    const double l = q < o ? X[(CT + o) * FBP + q] * ri : (q == o ? d : 0.0);
    if (i < nb && c < nb) {
      Lm[(size_t)(r0 + i) * n + r0 + c] = l;
      if (L32) L32[(size_t)(r0 + i) * np + r0 + c] = (float)l;
    }
  }
#pragma unroll
  for (int t = 0; t < CT / 4; ++t) {
    const int i = i0 + 4 * t;
    const double l = i > c ? u[t] : 0.0;
    if ((i ^ c) >= FB && i < nb && c < nb) {
      Lm[(size_t)(r0 + i) * n + r0 + c] = l;
      if (L32) L32[(size_t)(r0 + i) * np + r0 + c] = (float)l;
    }
    if (wout) wout[i * CT + c] = c > i ? u[t] : (c == i ? ri : 0.0);
  }
  if (tid == 0 && bad) atomicOr(&a.not_spd[lane], 1);
}

struct BlockSync {
  __device__ void operator()() const { __syncthreads(); }
};

// grid nlane, 256 threads: the first diagonal tile of every lane.  A later one
// is factored by the update launch that finishes it (the CTA that owns it).
__global__ void __launch_bounds__(256) chol_diag_kernel(KArgs a) {
  const int lane = blockIdx.x;
  if (lane >= a.nlane) return;
  const LaneDesc L = a.lanes[lane];
  const int n = 3 * a.tops[L.top].nmp;
  extern __shared__ __align__(16) double vec[];   // FD_VEC
  double acc[8][2];
  load_diag_tile(a.bd_L + L.bd0, n, 0, threadIdx.x, acc);
  factor_diag_tile(a, lane, a.bd_L + L.bd0, n, 0, acc, vec, threadIdx.x, BlockSync{});
}

// grid ((T - k - 1) 64 / RB, nlane), 256 threads: RB rows of row tile ti of
// the panel below the factored diagonal tile: X = A_ik L_kk^-T as an RB x 64
// x 64 FP64 product with the stored transposed inverse U_kk, upper triangular:
// column tile ct (8 columns) sums over m < 8 ct + 8, in increasing order.
// Stored in FP64 and, for the tensor-core update, split into TF32 hi / lo in
// the panel planes.  Loads and stores are row-contiguous.
// RB = 64: warp w has rows 8 w .. + 7; RB = 16: 8 rows and the column tiles q
// and 7 - q, the same work for every warp.
template <int RB>
__global__ void __launch_bounds__(256) chol_panel_kernel(KArgs a) {
  constexpr int SUB = CT / RB;
  const int lane = blockIdx.y;
  if (lane >= a.nlane) return;
  const LaneDesc L = a.lanes[lane];
  int n;
  const int T = lane_tiles(a, L, n), k = a.bd_kpanel;
  const int ti = k + 1 + blockIdx.x / SUB, rb = (blockIdx.x % SUB) * RB;   // first row in the tile
  if (ti >= T) return;   // rows below the diagonal tile: the panel is full (64 columns)
  const int r0 = k * CT, i0 = ti * CT + rb, mi = min(RB, n - i0);
  double *Lm = a.bd_L + L.bd0;
  extern __shared__ __align__(16) double dsm[];
  double *As = dsm, *Us = As + RB * CTP;
  const int tid = threadIdx.x, wp = tid >> 5, fr = (tid & 31) >> 2, fk = tid & 3;
  const double *w = a.bd_W + (size_t)lane * CT * CT;
#pragma unroll
  for (int q = 0; q < RB * CT / 256; ++q) {
    const int e = tid + 256 * q, r = e >> 6, c = e & 63;
    As[r * CTP + c] = (r < mi) ? Lm[(size_t)(i0 + r) * n + r0 + c] : 0.0;
  }
#pragma unroll
  for (int q = 0; q < CT * CT / 256; ++q) {
    const int e = tid + 256 * q;
    Us[(e >> 6) * CTP + (e & 63)] = w[e];
  }
  __syncthreads();
  constexpr int NT = RB == CT ? 8 : 2;   // column tiles of a warp
  double acc[NT][2];
#pragma unroll
  for (int t = 0; t < NT; ++t) acc[t][0] = acc[t][1] = 0.0;
  const int row = RB == CT ? 8 * wp + fr : 8 * (wp & 1) + fr;
  const int ct0 = RB == CT ? 0 : wp >> 1, ct1 = 7 - ct0;
  if (RB == CT) {
#pragma unroll
    for (int mb = 0; mb < 8; ++mb)
#pragma unroll
      for (int h = 0; h < 8; h += 4) {
        const int m = 8 * mb + h + fk;
        const double av = As[row * CTP + m];
#pragma unroll
        for (int t = mb; t < NT; ++t) mma8(acc[t], av, Us[m * CTP + 8 * t + fr]);
      }
  } else {
#pragma unroll 4
    for (int m = fk; m < 8 * ct1 + 8; m += 4) {
      const double av = As[row * CTP + m];
      if (m < 8 * ct0 + 8) mma8(acc[0], av, Us[m * CTP + 8 * ct0 + fr]);   // uniform: 4 divides the bound
      mma8(acc[1], av, Us[m * CTP + 8 * ct1 + fr]);
    }
  }
  __syncthreads();
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    const int ct = RB == CT ? t : (t ? ct1 : ct0);
    *(double2 *)&As[row * CTP + 8 * ct + 2 * fk] = make_double2(acc[t][0], acc[t][1]);
  }
  __syncthreads();
#pragma unroll 4
  for (int e = tid; e < RB * CT; e += 256) {
    const int r = e >> 6, c = e & 63;
    if (r < mi) {
      Lm[(size_t)(i0 + r) * n + r0 + c] = As[r * CTP + c];
      if (a.bd_tc) a.bd_L32[L.bd32 + (size_t)(i0 + r) * ((n + 3) & ~3) + r0 + c] = (float)As[r * CTP + c];
    }
  }
  if (a.bd_tc) {
    float *ph = a.bd_P + L.bdp0 + (size_t)(k & 1) * 2 * (T + 1) * PT + (size_t)ti * PT;
    float *pl = ph + (size_t)(T + 1) * PT;
#pragma unroll
    for (int q = 0; q < RB / 16; ++q) {
      const int e = tid + 256 * q, r = e % RB, g = e / RB, rt = rb + r;
      const double2 x01 = *(const double2 *)(As + r * CTP + 4 * g), x23 = *(const double2 *)(As + r * CTP + 4 * g + 2);
      float4 h, l;
      tf32_split(x01.x, h.x, l.x);
      tf32_split(x01.y, h.y, l.y);
      tf32_split(x23.x, h.z, l.z);
      tf32_split(x23.y, h.w, l.w);
      const int o = (rt >> 3) * 512 + g * 32 + (rt & 7) * 4;
      *(float4 *)(ph + o) = h;
      *(float4 *)(pl + o) = l;
    }
  }
}

// grid (nlane, tile pairs, parts), 256 threads: trailing tile (ti, tj),
// k < tj <= ti: A_ij -= L_ik L_jk^T in FP64.  B = 64: a CTA has the whole 64 x
// 64 tile (1 part), a warp 8 rows of it; B = 32: a quarter (4 parts), a warp 8
// rows of 16 columns.  The tile (k + 1, k + 1) belongs to one CTA either way,
// which factors it for the next panel.
template <int B>
__global__ void __launch_bounds__(256) chol_update_kernel(KArgs a) {
  constexpr int SUB = CT / B;
  const int lane = blockIdx.x;
  if (lane >= a.nlane) return;
  const LaneDesc L = a.lanes[lane];
  int n;
  const int T = lane_tiles(a, L, n), k = a.bd_kpanel;
  const int m = T - k - 1;
  const int p = blockIdx.y;
  if (m <= 0 || p >= m * (m + 1) / 2) return;
  int ii = (int)((sqrt(8.0 * p + 1.0) - 1.0) * 0.5);
  while (ii * (ii + 1) / 2 > p) --ii;
  while ((ii + 1) * (ii + 2) / 2 <= p) ++ii;
  const int jj = p - ii * (ii + 1) / 2;
  const int ti = k + 1 + ii, tj = k + 1 + jj, r0 = k * CT;
  const int qi = blockIdx.z / SUB, qj = blockIdx.z % SUB;
  double *Lm = a.bd_L + L.bd0;
  extern __shared__ __align__(16) double sh[];
  double *As = sh, *Bs = sh + CT * CTP;
  const int tid = threadIdx.x, w = tid >> 5, fr = (tid & 31) >> 2, fk = tid & 3;
  auto load = [&](double *dst, int i0, int rows) {   // rows i0 .. of the panel
#pragma unroll 8
    for (int e = tid; e < rows * CT; e += 256) {
      const int r = e >> 6, c = e & 63;
      dst[r * CTP + c] = (i0 + r < n) ? Lm[(size_t)(i0 + r) * n + r0 + c] : 0.0;
    }
  };
  if (p == 0) {
    if (blockIdx.z) return;
    load(As, ti * CT, CT);
    double acc[8][2];
    load_diag_tile(Lm, n, ti, tid, acc);
    __syncthreads();
    // rows beyond the matrix have zero panel rows: the identity stays
#pragma unroll 2
    for (int mm = fk; mm < CT; mm += 4) {
      const double av = -As[(8 * w + fr) * CTP + mm];
#pragma unroll
      for (int ct = 0; ct < 8; ++ct)
        if (ct <= w) mma8(acc[ct], av, As[(8 * ct + fr) * CTP + mm]);
    }
    factor_diag_tile(a, lane, Lm, n, ti, acc, sh, tid, BlockSync{});   // FD_VEC doubles fit the two tiles
    return;
  }
  if (ti == tj && qj > qi) return;
  const int i0 = ti * CT + qi * B, j0 = tj * CT + qj * B;
  load(As, i0, B);
  load(Bs, j0, B);
  constexpr int NT = B == CT ? 8 : 2;
  const int row = B == CT ? 8 * w + fr : 8 * (w >> 1) + fr, ct0 = B == CT ? 0 : 2 * (w & 1);
  double acc[NT][2];
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int i = i0 + row, c = j0 + 8 * (ct0 + t) + 2 * fk + q;
      acc[t][q] = (i < n && c < n) ? Lm[(size_t)i * n + c] : 0.0;
    }
  __syncthreads();
#pragma unroll 4
  for (int mm = fk; mm < CT; mm += 4) {
    const double av = -As[row * CTP + mm];
#pragma unroll
    for (int t = 0; t < NT; ++t) mma8(acc[t], av, Bs[(8 * (ct0 + t) + fr) * CTP + mm]);
  }
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int i = i0 + row, c = j0 + 8 * (ct0 + t) + 2 * fk + q;
      if (i < n && c < n) Lm[(size_t)i * n + c] = acc[t][q];
    }
}

// ------------------------------------------------------------ tensor cores
// Trailing updates on the 5th-generation tensor cores (mixed precision),
// two panels at a time.  For the panel pair (k, k + 1):
//   narrow: A_i,k+1 -= L_ik L_k+1,k^T for the column tile k + 1 (K = 64);
//   wide:   A_ij -= L_ik L_jk^T + L_i,k+1 L_j,k+1^T for j >= k + 2 (K = 128),
// so the FP64 trailing matrix is read and written once per two panels.
// L_ik = hi + lo is split into TF32 parts (the panel planes written by
// chol_panel_kernel, one slot per panel parity), the product taken as
// hi.hi + hi.lo + lo.hi (lo.lo is below FP32 rounding) and accumulated in
// FP32 in tensor memory; the FP64 tile subtracts it.  Diagonal tiles and
// panel solves stay in FP64.
//
// A CTA owns a 128-row block (row tiles ti, ti + 1) and up to UG column
// tiles of it, with one 64-column TMEM accumulator per column tile, and
// runs them as a pipeline of warp roles:
//   warp 0, one thread: bulk copies of the A block of each panel (the
//     second after the first panel's products are done) and of each B tile
//     (two shared-memory stages) from the panel planes;
//   warp 1, one thread: 24 tcgen05.mma (M 128, N 64, K 8) per column tile
//     and panel;
//   warps 2..9: epilogue, as soon as a tile's last panel is in: warp w
//     reads TMEM lanes 32 (w % 4) .. + 31 (rows) and column half (w - 2) / 4,
//     transposes the 32 x 32 block through its own shared-memory stage and
//     updates the FP64 rows with coalesced 256-byte accesses.
// The CTA whose first tile is the diagonal tile of the first updated column
// factors it afterwards (look-ahead for the next panel).  Every wait on a
// barrier is bounded; a wait that gives up flags the lane (not_spd bit 2,
// reported as a device-wait timeout) after the copies and products in
// flight are drained.
constexpr int UG = 8;                                 // column tiles per CTA (8 x 64 TMEM columns)
constexpr int U_A = 2 * 2 * CT * CT * 4;              // A hi + lo, 128 rows, one panel
constexpr int U_B = 2 * CT * CT * 4;                  // one B stage, hi + lo
constexpr int U_STG = 32 * 33 * 4;                    // epilogue transpose stage per warp
constexpr int U_SMEM = U_A + 2 * U_B + 8 * U_STG;
constexpr int U_THREADS = 320;
constexpr uint32_t U_WAIT_NS = 100000;                // suspend hint per poll
constexpr uint32_t U_WAIT_MAX = 20000;                // polls: about 2 s at most

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// UMMA shared-memory descriptor: start >> 4 [0,14), LBO >> 4 [16,30),
// SBO >> 4 [32,46), version 1 [46,48), no swizzle (layout type 0 [61,64)).
// K-major without swizzle: LBO = byte step between the two K-adjacent core
// matrices of one K = 8 slice, SBO = byte step between 8-row groups.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  for (uint32_t it = 0; it < U_WAIT_MAX; ++it) {
    uint32_t done;
    asm volatile("{\n\t.reg .pred P1;\n\tmbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2, %3;\n\t"
                 "selp.b32 %0, 1, 0, P1;\n\t}\n"
                 : "=r"(done)
                 : "r"(bar), "r"(parity), "r"(U_WAIT_NS)
                 : "memory");
    if (done) return true;
  }
  return false;
}

__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// panel planes of panel kp of a lane: hi, then lo (T + 1 tiles each)
__device__ __forceinline__ const float *plane_hi(const KArgs &a, const LaneDesc &L, int T, int kp) {
  return a.bd_P + L.bdp0 + (size_t)(kp & 1) * 2 * (T + 1) * PT;
}

// One CTA per work item (lane << 16 | R << 8 | g) of the launch (bd_update_items):
// narrow (nph = 1): column tile k + 1 only, panel k; wide (nph = 2): column
// tiles >= k + 2, panels k and k + 1.  U_THREADS threads, one CTA per SM.
__global__ void __launch_bounds__(U_THREADS, 1) chol_update_tc_kernel(KArgs a, const int *items, int nph, int ug) {
  const int item = items[blockIdx.x];
  const int lane = item >> 16, R = (item >> 8) & 255, g = item & 255;
  const LaneDesc L = a.lanes[lane];
  int n;
  const int T = lane_tiles(a, L, n), k = a.bd_kpanel;
  const int cf = k + nph;   // first updated row and column tile
  const int m = T - cf;
  if (m <= 0 || 2 * R >= m) return;   // not produced by the item tables; uniform over the CTA
  const int ncol = nph == 1 ? 1 : min(2 * R + 2, m), c0 = g * ug;   // ug <= UG
  if (c0 >= ncol) return;
  const int nt = min(ug, ncol - c0);
  const int ti0 = cf + 2 * R, tj0 = cf + c0;
  double *Lm = a.bd_L + L.bd0;

  extern __shared__ __align__(1024) unsigned char tsm[];
  unsigned char *base = (unsigned char *)(((uintptr_t)tsm + 1023) & ~(uintptr_t)1023);
  const uint32_t s_ahi = smem_u32(base), s_alo = s_ahi + U_A / 2;
  const uint32_t s_b0 = s_ahi + U_A;   // stage s: hi at s_b0 + s U_B, lo 16 KB later
  // fullA, fullB0/1, emptyB0/1, afree, mdone, tfull0..7
  __shared__ __align__(8) uint64_t bars[7 + UG];
  __shared__ uint32_t tmem_slot;
  __shared__ int gaveup;
  const uint32_t b_fullA = smem_u32(&bars[0]), b_fullB = smem_u32(&bars[1]), b_emptyB = smem_u32(&bars[3]);
  const uint32_t b_afree = smem_u32(&bars[5]), b_mdone = smem_u32(&bars[6]), b_tfull = smem_u32(&bars[7]);
  const int tid = threadIdx.x, warp = tid >> 5, lid = tid & 31;
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"(UG * CT));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int q = 0; q < 7 + UG; ++q)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bars[q])));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    gaveup = 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t taddr = tmem_slot;

  if (warp == 0) {
    if (lid == 0) {
      bool ok = true;
      int last[2] = {-1, -1};
      for (int p = 0; p < nph && ok; ++p) {
        const float *ph = plane_hi(a, L, T, k + p), *pl = ph + (size_t)(T + 1) * PT;
        // the second panel's A block replaces the first once its products are done
        if (p == 1 && !mbar_wait(b_afree, 0)) { ok = false; break; }
        mbar_expect(b_fullA, U_A);
        bulk_load(s_ahi, ph + (size_t)ti0 * PT, U_A / 2, b_fullA);
        bulk_load(s_alo, pl + (size_t)ti0 * PT, U_A / 2, b_fullA);
        for (int t = 0; t < nt; ++t) {
          const int u = p * nt + t, s = u & 1;
          if (u >= 2 && !mbar_wait(b_emptyB + 8 * s, ((u >> 1) - 1) & 1)) { ok = false; break; }
          const uint32_t dst = s_b0 + (uint32_t)s * U_B;
          mbar_expect(b_fullB + 8 * s, U_B);
          bulk_load(dst, ph + (size_t)(tj0 + t) * PT, U_B / 2, b_fullB + 8 * s);
          bulk_load(dst + U_B / 2, pl + (size_t)(tj0 + t) * PT, U_B / 2, b_fullB + 8 * s);
          last[s] = u;
        }
      }
      // drain: no copy may still be writing shared memory when the CTA ends
      // (the last A load has phase parity nph - 1; the MMA thread waited
      // for the earlier one)
      ok = mbar_wait(b_fullA, (nph - 1) & 1) && ok;
      for (int s = 0; s < 2; ++s)
        if (last[s] >= 0) ok = mbar_wait(b_fullB + 8 * s, (last[s] >> 1) & 1) && ok;
      if (!ok) gaveup = 1;
    }
  } else if (warp == 1) {
    if (lid == 0) {
      // kind::tf32, D F32 [4,6) = 1, A TF32 [7,10) = 2, B TF32 [10,13) = 2,
      // both K-major, N >> 3 at [17,23), M >> 4 at [24,29)
      const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(CT >> 3) << 17) |
                             ((uint32_t)(2 * CT >> 4) << 24);
      bool ok = true;
      for (int p = 0; p < nph && ok; ++p) {
        if (!mbar_wait(b_fullA, p & 1)) { ok = false; break; }
        for (int t = 0; t < nt; ++t) {
          const int u = p * nt + t, s = u & 1;
          if (!mbar_wait(b_fullB + 8 * s, (u >> 1) & 1)) { ok = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t bhi = s_b0 + (uint32_t)s * U_B, blo = bhi + U_B / 2;
          const uint32_t dacc = taddr + (uint32_t)(t * CT);
          for (int ks = 0; ks < CT / 8; ++ks) {
            for (int pp = 0; pp < 3; ++pp) {
              const uint32_t sa = (pp == 2 ? s_alo : s_ahi) + (uint32_t)ks * 256u;
              const uint32_t sb = (pp == 1 ? blo : bhi) + (uint32_t)ks * 256u;
              const uint64_t da = umma_desc(sa, 128, 2048), db = umma_desc(sb, 128, 2048);
              const uint32_t acc = (p | ks | pp) ? 1u : 0u;
              asm volatile(
                  "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                  "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}\n"
                  :: "r"(dacc), "l"(da), "l"(db), "r"(idesc), "r"(acc));
            }
          }
          umma_commit(b_emptyB + 8 * s);
          if (p == nph - 1) umma_commit(b_tfull + 8 * t);
        }
        if (ok && p == 0 && nph > 1) umma_commit(b_afree);
      }
      // every product issued by this thread has landed before TMEM is freed
      umma_commit(b_mdone);
      ok = mbar_wait(b_mdone, 0) && ok;
      if (!ok) gaveup = 1;
    }
  } else {
    const int e = warp - 2, q = warp & 3, h = e >> 2;
    float *stg = (float *)(base + U_A + 2 * U_B + e * U_STG);
    uint32_t eok = 1;
    for (int t = 0; t < nt; ++t) {
      const int tj = tj0 + t, col = tj * CT + h * 32 + lid;
      // the tile's FP64 elements while its products are on their way, and the
      // next tile's lines towards L2: a tile's time was that of its loads,
      // issued after the wait (4.2 us a tile of the widest launch; now 3.6)
      double old[32];
#pragma unroll
      for (int rr = 0; rr < 32; ++rr) {
        const int rw = q * 32 + rr, trow = ti0 + (rw >> 6), grow = trow * CT + (rw & 63);
        old[rr] = (grow < n && col < n && trow >= tj) ? Lm[(size_t)grow * n + col] : 0.0;
      }
      if (t + 1 < nt) {
        const int rw = q * 32 + lid, trow = ti0 + (rw >> 6), grow = trow * CT + (rw & 63), c0 = (tj + 1) * CT + h * 32;
        if (grow < n && c0 + 31 < n && trow > tj) {
          const double *next = Lm + (size_t)grow * n + c0;
          asm volatile("prefetch.global.L2 [%0];" ::"l"(next));
          asm volatile("prefetch.global.L2 [%0];" ::"l"(next + 16));
          asm volatile("prefetch.global.L2 [%0];" ::"l"(next + 31));
        }
      }
      const bool ok = __all_sync(0xffffffffu, mbar_wait(b_tfull + 8 * t, 0));
      if (!ok) {
        if (lid == 0) gaveup = 1;
        eok = 0;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      uint32_t v[32];
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
          "%14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
          : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
            "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
            "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]),
            "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]),
            "=r"(v[30]), "=r"(v[31])
          : "r"(taddr + ((uint32_t)(q * 32) << 16) + (uint32_t)(t * CT + h * 32)));
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      // lane = row of the TMEM block: transpose so that a lane owns a column
#pragma unroll
      for (int c = 0; c < 32; ++c) stg[lid * 33 + c] = __uint_as_float(v[c]);
      __syncwarp();
#pragma unroll
      for (int rr = 0; rr < 32; ++rr) {
        const int rw = q * 32 + rr, trow = ti0 + (rw >> 6), grow = trow * CT + (rw & 63);
        if (grow < n && col < n && trow >= tj) Lm[(size_t)grow * n + col] = old[rr] - (double)stg[rr * 33 + lid];
      }
      __syncwarp();
    }
    if (R == 0 && g == 0) {
      // tile (cf, cf), updated above by this CTA, is final: the eight
      // epilogue warps factor it for the next panel (the operand area is
      // free: every product has been read out of TMEM)
      const auto esync = [] { asm volatile("bar.sync 1, 256;" ::: "memory"); };
      uint32_t all_ok;   // the same on all eight warps
      asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.and.pred p, 1, 256, q;\n\t"
                   "selp.u32 %0, 1, 0, p;\n\t}\n"
                   : "=r"(all_ok)
                   : "r"(eok)
                   : "memory");
      if (all_ok) {
        double acc[8][2];
        load_diag_tile(Lm, n, cf, tid - 64, acc);
        factor_diag_tile(a, lane, Lm, n, cf, acc, (double *)base, tid - 64, esync);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(UG * CT));
  }
  if (tid == 0 && gaveup) atomicOr(&a.not_spd[lane], 2);   // a tensor-core pipeline wait gave up
}

// ------------------------------------------------------------ step
// grid (ceil(maxN / 128), nlane): xi of every bead
__global__ void __launch_bounds__(128) bd_noise_kernel(KArgs a) {
  const int lane = blockIdx.y;
  if (lane >= a.nlane) return;
  const LaneDesc L = a.lanes[lane];
  const int N = a.tops[L.top].nmp;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  double n0, n1, n2;
  noise3(a, lane, L, i, a.bd_istep, a.noise_base, n0, n1, n2);
  double *xi = a.bd_xi + 3 * (size_t)(L.state0 + i);
  xi[0] = n0; xi[1] = n1; xi[2] = n2;
}

// grid (ceil(maxN * 3 / (8 R)), nlane), 256 threads: one warp per R rows k of
// the lane: dx_k = rlan1 sum_c D_kc F_c + rlan2 sum_{c <= k} L_kc xi_c, x += dx.
// HBM-bound: the mixed-precision path streams FP32 copies of D and L
// (products and sums in FP64), the FP64 path the FP64 matrices.  A group of
// four columns costs 4 cycles of L1 for a row's elements but 32 for its F (four
// doubles per lane, 32 bytes apart), so with one row per warp L1 was the bound
// (640 MB in 187 us, 3.4 TB/s; 32 lanes of 100 to 1000 beads).  R = 4 rows share
// the loads of F and xi, and the matrices stream past L1 with 16 float4 in flight
// per lane: 111 us (5.8 TB/s; more rows, warps or bytes in flight, or rows
// staged by bulk copies, were no faster).  Every row's sum has the same order
// for either R (columns by lane, then a butterfly).
struct Rows64 {
  const double *D, *L;
  size_t stride;
};
struct Rows32 {   // rows padded to a multiple of 4 (16-byte aligned)
  const float *D, *L;
  size_t stride;
};

template <int R>
__device__ __forceinline__ void row_dots(const Rows64 &m, const double *F, const double *xi, int n, int k0, int lid,
                                         double (&df)[R], double (&dr)[R]) {
  const double *D[R], *L[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const size_t o = (size_t)min(k0 + r, n - 1) * m.stride;
    D[r] = m.D + o;
    L[r] = m.L + o;
  }
  int c = lid;
#pragma unroll 4
  for (; c <= k0; c += 32) {   // L: columns up to k0 for all rows
    const double f = F[c], x = xi[c];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      df[r] = fma(D[r][c], f, df[r]);
      dr[r] = fma(L[r][c], x, dr[r]);
    }
  }
#pragma unroll 4
  for (; c < n; c += 32) {
    const double f = F[c];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      df[r] = fma(D[r][c], f, df[r]);
      if (r > 0 && c <= k0 + r) dr[r] = fma(L[r][c], xi[c], dr[r]);
    }
  }
}

// float4 loads for the whole 4-column groups inside the matrix, then the < 4
// last columns; k0 is a multiple of R
template <int R>
__device__ __forceinline__ void row_dots(const Rows32 &m, const double *F, const double *xi, int n, int k0, int lid,
                                         double (&df)[R], double (&dr)[R]) {
  const float4 *D4[R], *L4[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const size_t o = (size_t)min(k0 + r, n - 1) * m.stride;
    D4[r] = (const float4 *)(m.D + o);
    L4[r] = (const float4 *)(m.L + o);
  }
  const int n4 = n >> 2;
  // L is zero above the diagonal: whole groups up to the rows' own columns
  const int k4 = min((k0 >> 2) + 1, n4);
  auto dot4 = [](const float4 &e, const double *v, double s) {
    return fma((double)e.w, v[3], fma((double)e.z, v[2], fma((double)e.y, v[1], fma((double)e.x, v[0], s))));
  };
  int g = lid;
#pragma unroll 2
  for (; g < k4; g += 32) {
    float4 d[R], l[R];
#pragma unroll
    for (int r = 0; r < R; ++r) d[r] = __ldcs(&D4[r][g]);
#pragma unroll
    for (int r = 0; r < R; ++r) l[r] = __ldcs(&L4[r][g]);
    const double f[4] = {F[4 * g], F[4 * g + 1], F[4 * g + 2], F[4 * g + 3]};
    const double x[4] = {xi[4 * g], xi[4 * g + 1], xi[4 * g + 2], xi[4 * g + 3]};
#pragma unroll
    for (int r = 0; r < R; ++r) {
      df[r] = dot4(d[r], f, df[r]);
      dr[r] = dot4(l[r], x, dr[r]);
    }
  }
#pragma unroll 4
  for (; g < n4; g += 32) {
    const double f[4] = {F[4 * g], F[4 * g + 1], F[4 * g + 2], F[4 * g + 3]};
#pragma unroll
    for (int r = 0; r < R; ++r) df[r] = dot4(__ldcs(&D4[r][g]), f, df[r]);
  }
  const int c = 4 * n4 + lid;
  if (c < n) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      df[r] = fma((double)((const float *)D4[r])[c], F[c], df[r]);
      if (c <= k0 + r) dr[r] = fma((double)((const float *)L4[r])[c], xi[c], dr[r]);
    }
  }
}

template <int R>
__global__ void __launch_bounds__(256, 2) bd_update_kernel(KArgs a) {
  const int lane = blockIdx.y;
  if (lane >= a.nlane) return;
  const LaneDesc L = a.lanes[lane];
  const int n = 3 * a.tops[L.top].nmp;
  const int warp = threadIdx.x >> 5, lid = threadIdx.x & 31;
  const int k0 = (blockIdx.x * 8 + warp) * R;
  if (blockIdx.x == 0 && threadIdx.x == 0) a.lstate[lane].istep = a.bd_istep;
  if (k0 >= n) return;
  const double *F = a.bd_F + 3 * (size_t)L.state0, *xi = a.bd_xi + 3 * (size_t)L.state0;
  double df[R], dr[R];
#pragma unroll
  for (int r = 0; r < R; ++r) df[r] = dr[r] = 0.0;
  if (a.bd_tc) {
    const int np = (n + 3) & ~3;
    row_dots<R>(Rows32{a.bd_D32 + L.bd32, a.bd_L32 + L.bd32, (size_t)np}, F, xi, n, k0, lid, df, dr);
    if (a.bd_refine) {   // - (E z)_k / 2
      const double *z = a.bd_z + 3 * (size_t)L.state0;
      const int n4 = n >> 2;
#pragma unroll 1
      for (int r = 0; r < R; ++r) {
        const size_t row = L.bd32 + (size_t)min(k0 + r, n - 1) * np;
        const float4 *E4 = (const float4 *)(a.bd_E32 + row);
        double ez = 0.0;
        for (int g = lid; g < n4; g += 32) {
          const float4 e = E4[g];
          ez += (double)e.x * z[4 * g] + (double)e.y * z[4 * g + 1] + (double)e.z * z[4 * g + 2] + (double)e.w * z[4 * g + 3];
        }
        if (lid < n - 4 * n4) ez += (double)a.bd_E32[row + 4 * n4 + lid] * z[4 * n4 + lid];
#pragma unroll
        for (int q = 0; q < R; ++q)
          if (q == r) dr[q] -= 0.5 * ez;
      }
    }
  } else {
    row_dots<R>(Rows64{a.bd_D + L.bd0, a.bd_L + L.bd0, (size_t)n}, F, xi, n, k0, lid, df, dr);
  }
  double mf = 0.0, mr = 0.0;   // lane r: row k0 + r
#pragma unroll
  for (int r = 0; r < R; ++r) {
    for (int o = 16; o > 0; o >>= 1) {
      df[r] += __shfl_xor_sync(0xffffffffu, df[r], o);
      dr[r] += __shfl_xor_sync(0xffffffffu, dr[r], o);
    }
    if (lid == r) {
      mf = df[r];
      mr = dr[r];
    }
  }
  if (lid < R && k0 + lid < n) {
    const double T = a.lab_T[a.lstate[lane].label];
    const double rl1 = a.tstep / (a.boltz * T), rl2 = sqrt(2.0 * a.tstep);
    const double dx = rl1 * mf + rl2 * mr;
    const size_t o = 3 * (size_t)L.state0 + k0 + lid;
    a.xyz[o] += dx;
    a.pxyz[o] += dx;
    a.dxyz[o] += dx;
  }
}

// ------------------------------------------------------------ refinement
// The mixed-precision step samples L xi with the FP32 factor L, whose
// L L^T = D + E differs from D by the rounding of the split-TF32 updates and
// of the FP32 copy (|E| ~ 1e-7 |D|).  M = L - E L^-T / 2 has
// M M^T = D + E L^-T L^-1 E / 4, so the step samples M xi = L xi - E z / 2
// with z = L^-T xi.  E is formed at each refresh with FP64 sums; z and E z
// are FP32 data with FP64 sums (errors of order 1e-7 of a 1e-7 correction).
constexpr int RT = 64;
constexpr int RT_SMEM = 2 * RT * (RT + 1) * (int)sizeof(double);

// grid (Tmax (Tmax + 1) / 2, nlane), 256 threads: tile (I, J), I >= J, of
// E = L L^T - D in FP64, written to both halves of the FP32 E
__global__ void __launch_bounds__(256) refine_residual_kernel(KArgs a) {
  const int lane = blockIdx.y;
  if (lane >= a.nlane) return;
  const LaneDesc L = a.lanes[lane];
  const int n = 3 * a.tops[L.top].nmp, T = (n + RT - 1) / RT, ld = (n + 3) & ~3;
  const int p = blockIdx.x;
  if (p >= T * (T + 1) / 2) return;
  int I = (int)((sqrt(8.0 * p + 1.0) - 1.0) * 0.5);
  while ((I + 1) * (I + 2) / 2 <= p) ++I;
  while (I * (I + 1) / 2 > p) --I;
  const int J = p - I * (I + 1) / 2;
  extern __shared__ double rsm[];
  double *As = rsm, *Bs = rsm + RT * (RT + 1);
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  double acc[4][4];
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int w = 0; w < 4; ++w) acc[q][w] = 0.0;
  const float *Lm = a.bd_L32 + L.bd32;
  for (int K = 0; K <= J; ++K) {   // L_IK L_JK^T; L is zero above its diagonal
    for (int e = threadIdx.x; e < RT * RT; e += 256) {
      const int r = e / RT, c = e - r * RT, gc = K * RT + c, ra = I * RT + r, rb = J * RT + r;
      As[r * (RT + 1) + c] = (ra < n && gc < n) ? (double)Lm[(size_t)ra * ld + gc] : 0.0;
      Bs[r * (RT + 1) + c] = (rb < n && gc < n) ? (double)Lm[(size_t)rb * ld + gc] : 0.0;
    }
    __syncthreads();
    // thread (ty, tx): rows ty * 4 + q, columns tx + 16 w (consecutive tx
    // read rows 65 doubles apart: no shared-memory bank conflicts)
    for (int k = 0; k < RT; ++k) {
      double av[4], bv[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) { av[q] = As[(ty * 4 + q) * (RT + 1) + k]; bv[q] = Bs[(tx + 16 * q) * (RT + 1) + k]; }
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int w = 0; w < 4; ++w) acc[q][w] = fma(av[q], bv[w], acc[q][w]);
    }
    __syncthreads();
  }
  const double *D = a.bd_D64 + L.bd0;
  float *E = a.bd_E32 + L.bd32;
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const int row = I * RT + ty * 4 + q, col = J * RT + tx + 16 * w;
      if (row < n && col < n) {
        const float e = (float)(acc[q][w] - D[(size_t)row * n + col]);
        E[(size_t)row * ld + col] = e;
        if (I != J) E[(size_t)col * ld + row] = e;
      }
    }
}

// grid (Tmax, nlane), 64 threads: W_b = inverse of the diagonal tile L_bb of
// the FP32 factor (FP64 forward substitution, one column per thread; rows
// past n act as the identity)
__global__ void __launch_bounds__(64) refine_inverse_kernel(KArgs a) {
  const int lane = blockIdx.y;
  if (lane >= a.nlane) return;
  const LaneDesc L = a.lanes[lane];
  const int n = 3 * a.tops[L.top].nmp, T = (n + RT - 1) / RT, ld = (n + 3) & ~3;
  const int b = blockIdx.x;
  if (b >= T) return;
  extern __shared__ double inv_buf[];   // L_bb, then its inverse (RT_SMEM bytes)
  double *Lt = inv_buf, *X = inv_buf + RT * (RT + 1);
  const float *Lm = a.bd_L32 + L.bd32;
  const int c = threadIdx.x;
  for (int r = 0; r < RT; ++r) {
    const int gr = b * RT + r, gc = b * RT + c;
    Lt[r * (RT + 1) + c] = (gr < n && gc < n) ? (double)Lm[(size_t)gr * ld + gc] : (r == c ? 1.0 : 0.0);
  }
  __syncthreads();
  for (int i = 0; i < RT; ++i) {
    double x = 0.0;
    if (i >= c) {
      double s = (i == c) ? 1.0 : 0.0;
      for (int k = c; k < i; ++k) s -= Lt[i * (RT + 1) + k] * X[k * (RT + 1) + c];
      x = s / Lt[i * (RT + 1) + i];
    }
    X[i * (RT + 1) + c] = x;
  }
  float *W = a.bd_W32 + L.bdw0 + (size_t)b * RT * RT;
  for (int i = 0; i < RT; ++i) W[i * RT + c] = (float)X[i * (RT + 1) + c];
}

// grid nlane, 1024 threads: z = L^-T xi by blocked back substitution from
// the last tile: rhs_b = xi_b - sum over the rows below of L^T z, then
// z_b = W_b^T rhs_b
constexpr int TRSV_THREADS = 1024;
__global__ void __launch_bounds__(TRSV_THREADS) refine_trsv_kernel(KArgs a) {
  const int lane = blockIdx.x;
  if (lane >= a.nlane) return;
  const LaneDesc L = a.lanes[lane];
  const int n = 3 * a.tops[L.top].nmp, T = (n + RT - 1) / RT, ld = (n + 3) & ~3;
  extern __shared__ double trsm_buf[];
  double *zs = trsm_buf;                         // n
  double *part = trsm_buf + ((n + 1) & ~1);      // 16 x 64
  double *rhs = part + 16 * RT;             // 64
  const float *Lm = a.bd_L32 + L.bd32;
  const double *xi = a.bd_xi + 3 * (size_t)L.state0;
  const int c = threadIdx.x & (RT - 1), g = threadIdx.x >> 6;
  for (int b = T - 1; b >= 0; --b) {
    const int j = b * RT + c;
    double sacc = 0.0;
    if (j < n)
      for (int r = (b + 1) * RT + g; r < n; r += 16) sacc += (double)Lm[(size_t)r * ld + j] * zs[r];
    part[g * RT + c] = sacc;
    __syncthreads();
    if (threadIdx.x < RT) {
      double t = 0.0;
      for (int q = 0; q < 16; ++q) t += part[q * RT + c];
      rhs[c] = (j < n) ? xi[j] - t : 0.0;
    }
    __syncthreads();
    if (threadIdx.x < RT) {
      const float *W = a.bd_W32 + L.bdw0 + (size_t)b * RT * RT;
      double z = 0.0;
      for (int i = c; i < RT; ++i) z += (double)W[i * RT + c] * rhs[i];
      if (j < n) zs[j] = z;
    }
    __syncthreads();
  }
  double *zo = a.bd_z + 3 * (size_t)L.state0;
  for (int k = threadIdx.x; k < n; k += TRSV_THREADS) zo[k] = zs[k];
}

// grid (ceil(maxN / 8), nlane), 256 threads: one warp per bead sums its FENE
// and WCA records (force_fene.F90, force_wca.F90) in record order
__global__ void __launch_bounds__(256) bd_force_kernel(KArgs a) {
  const int lane = blockIdx.y;
  if (lane >= a.nlane) return;
  const LaneDesc L = a.lanes[lane];
  const TopDesc T = a.tops[L.top];
  const int warp = threadIdx.x >> 5, lid = threadIdx.x & 31;
  const int i = blockIdx.x * 8 + warp;
  if (i >= T.nmp) return;
  const double *x = a.xyz + 3 * (size_t)L.state0;
  const int p0 = a.bd_ptr[T.bp0 + i], p1 = a.bd_ptr[T.bp0 + i + 1];
  const double xi0 = x[3 * i], xi1 = x[3 * i + 1], xi2 = x[3 * i + 2];
  double fx = 0.0, fy = 0.0, fz = 0.0;
  int nclamp = 0;
  const double far = a.wca_rcut2 * (1.0 - 1e-12);   // nat2 / dist2 is below the cutoff ratio whatever the rounding
  // entry (j, class * 2 + kind): the record's force on i is f (x_i - x_j),
  // the same numbers as -/+ f (x_i2 - x_i1) in the record's own orientation.
  // A lane's entries, four at a time: entries, then positions and classes,
  // are in flight together (one at a time each waited for its own two loads)
  constexpr int U = 4;
  int2 nx[U];   // the next four
  auto fetch = [&](int pb) {
#pragma unroll
    for (int u = 0; u < U; ++u) nx[u] = pb + 32 * u < p1 ? __ldcs(&a.bd_ent[T.be0 + pb + 32 * u]) : make_int2(-1, 0);
  };
  fetch(p0 + lid);
  for (int pb = p0 + lid; pb < p1; pb += 32 * U) {
    int2 e[U];
    double v[U][3], dist2[U], nat[U];
#pragma unroll
    for (int u = 0; u < U; ++u) e[u] = nx[u];
    fetch(pb + 32 * U);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int j = max(e[u].x, 0);
      v[u][0] = xi0 - x[3 * j];
      v[u][1] = xi1 - x[3 * j + 1];
      v[u][2] = xi2 - x[3 * j + 2];
      nat[u] = ((e[u].y & 1) ? a.wca_cls : a.fene_cls)[3 * (size_t)(e[u].y >> 1)];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) dist2[u] = v[u][0] * v[u][0] + v[u][1] * v[u][1] + v[u][2] * v[u][2];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int cl = e[u].y >> 1;
      if (e[u].x < 0) continue;
      double f;
      if (!(e[u].y & 1)) {
        const double *pc = a.fene_cls + 3 * (size_t)cl;   // nat, coef, dist2
        const double dist = sqrt(dist2[u]);
        const double dd = dist - nat[u];
        f = -pc[1] * dd / (1.0 - dd * dd / pc[2]) / dist;
      } else {
        const double *pc = a.wca_cls + 3 * (size_t)cl;    // nat, coef rep, coef att
        const double nat2 = nat[u] * nat[u];
        if (nat2 < far * dist2[u]) continue;   // most pairs: no division
        const double ro2 = nat2 / dist2[u];
        if (ro2 < a.wca_rcut2) continue;
        const double ro4 = ro2 * ro2, ro8 = ro4 * ro4, ro14 = ro8 * ro4 * ro2;
        const double coef = (ro2 > 1.0) ? pc[1] : pc[2];
        f = 12.0 * coef / nat2 * (ro14 - ro8);
        if (f > 50.0) { f = 50.0; nclamp += e[u].x > i; }   // DE_MAX; the record is counted once, from its lower bead
      }
      fx += f * v[u][0]; fy += f * v[u][1]; fz += f * v[u][2];
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    fx += __shfl_xor_sync(0xffffffffu, fx, o);
    fy += __shfl_xor_sync(0xffffffffu, fy, o);
    fz += __shfl_xor_sync(0xffffffffu, fz, o);
    nclamp += __shfl_xor_sync(0xffffffffu, nclamp, o);
  }
  if (lid == 0) {
    double *F = a.bd_F + 3 * (size_t)(L.state0 + i);
    F[0] = fx; F[1] = fy; F[2] = fz;
    if (nclamp) atomicAdd((unsigned long long *)&a.lstate[lane].nclamp, (unsigned long long)nclamp);
  }
}

// pivot_rcp and CUDA's reciprocal of n numbers, for its test
__global__ void pivot_rcp_kernel(const double *p, int n, double *own, double *cuda) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) { own[i] = pivot_rcp(p[i]); cuda[i] = __drcp_rn(p[i]); }
}
cudaError_t pivot_rcp_launch(const double *p, int n, double *own, double *cuda) {
  pivot_rcp_kernel<<<(n + 255) / 256, 256>>>(p, n, own, cuda);
  return cudaGetLastError();
}

// ------------------------------------------------------------ launches
// Work items of the tensor-core updates (lane << 16 | R << 8 | g): for the
// panel pair starting at k (k even) the narrow launch's items are
// items[koff[k] .. koff[k + 1]) and the wide launch's items[koff[k + 1] ..
// koff[k + 2]).  Items that factor the next diagonal tile come first, the
// rest by decreasing tile count.  lane_T = tiles per lane.
// kug[i]: column tiles per item of launch i.  UG of them share one load of the
// 128 rows' operands, but the chip has 148 CTAs and a launch lasts as long as
// its last item: the size with the shortest time at U_ITEM us per item, U_TILE
// per column tile and U_DIAG for the diagonal tile.  With 8 tiles per item
// always, the last ten wide launches of 32 chains of 100 to 1,000 beads took
// 40 us each, with 1 to 4 they take 22 (a launch of the diagonal tile alone:
// 20).
void bd_update_items(const std::vector<int> &lane_T, std::vector<int> &items, std::vector<int> &koff,
                     std::vector<int> &kug) {
  constexpr double U_ITEM = 5.0, U_TILE = 3.5, U_DIAG = 10.0;
  int tmax = 0;
  for (int t : lane_T) tmax = std::max(tmax, t);
  items.clear();
  koff.assign(1, 0);
  kug.clear();
  for (int k = 0; k < tmax + 1; ++k) {
    const int nph = (k & 1) ? 2 : 1;   // odd entries: the wide launch of the pair starting at k - 1
    const int kp = k & ~1;
    std::vector<std::pair<int, int>> best;   // (order key, item)
    double best_time = 0.0;
    int best_ug = UG;
    for (int ug = UG; ug >= (nph == 1 ? UG : 1); ug >>= 1) {
      if (ug < UG && tmax > 255 * ug) break;   // g has 8 bits
      std::vector<std::pair<int, int>> ks;
      double sum = 0.0, longest = 0.0;
      for (size_t l = 0; l < lane_T.size(); ++l) {
        const int m = lane_T[l] - kp - nph;
        for (int R = 0; 2 * R < m; ++R) {
          const int ncol = nph == 1 ? 1 : std::min(2 * R + 2, m);
          for (int g = 0; g * ug < ncol; ++g) {
            const int nt = std::min(ug, ncol - g * ug);
            const bool first = R == 0 && g == 0;   // factors the next diagonal tile
            ks.push_back({(first ? 1 << 20 : 0) + nt, (int)(l << 16) | (R << 8) | g});
            const double t = U_ITEM + nt * U_TILE + (first ? U_DIAG : 0.0);
            sum += t;
            longest = std::max(longest, t);
          }
        }
      }
      // the longest come first, so the rest fills up behind them
      const double time = std::max(longest, sum / BD_SMS + 0.5 * (U_ITEM + ug * U_TILE));
      if (best.empty() || time < best_time) {
        best.swap(ks);
        best_time = time;
        best_ug = ug;
      }
    }
    std::stable_sort(best.begin(), best.end(), [](const std::pair<int, int> &x, const std::pair<int, int> &y) {
      return x.first > y.first;
    });
    for (auto &e : best) items.push_back(e.second);
    koff.push_back((int)items.size());
    kug.push_back(best_ug);
  }
}

// Panel launch: 64 rows per CTA, or 16 while the 64-row CTAs would leave SMs
// idle (a panel is FP64-bound, so splitting the rows divides its time, but
// every CTA reads U again); the FP64 update's quarter tiles follow the same
// line.  A step with refresh, small against large blocks: 150 beads 167 / 177
// us, 8 x 150 186 / 193, 16 x 150 226 / 227, 32 x 150 301 / 302, 400 beads 405 /
// 418; mixed 400 beads 500 / 531, 16 x 400 794 / 805.
cudaError_t panel_launch(cudaStream_t st, const KArgs &a, int m) {
  if ((long long)m * a.nlane <= BD_SMS)
    chol_panel_kernel<16><<<dim3(4 * m, a.nlane), 256, (16 + CT) * CTP * sizeof(double), st>>>(a);
  else
    chol_panel_kernel<CT><<<dim3(m, a.nlane), 256, U64_SMEM, st>>>(a);
  return cudaGetLastError();
}

cudaError_t bd_refactor_launch(cudaStream_t st, KArgs a, int max_nmp, const int *items, const int *koff,
                               const int *kug) {
  cudaError_t e = cudaFuncSetAttribute(chol_diag_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FD_VEC * sizeof(double));
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(chol_update_kernel<CT>, cudaFuncAttributeMaxDynamicSharedMemorySize, U64_SMEM);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(chol_update_kernel<CT / 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, U64_SMEM);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(chol_panel_kernel<CT>, cudaFuncAttributeMaxDynamicSharedMemorySize, U64_SMEM);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(chol_update_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, U_SMEM + 1024);
  if (e != cudaSuccess) return e;
  if (a.bd_tc && (!a.bd_P || !items || !koff || !kug)) return cudaErrorInvalidValue;
  const long long nn = (long long)max_nmp * max_nmp;
  rpy_kernel<<<dim3((unsigned)((nn + 255) / 256), a.nlane), 256, 0, st>>>(a);
  chol_diag_kernel<<<a.nlane, 256, FD_VEC * sizeof(double), st>>>(a);
  const int T = (3 * max_nmp + CT - 1) / CT;
  if (a.bd_tc) {
    // panel pairs: panel k, narrow update (column k + 1), panel k + 1, wide update
    for (int k = 0; k + 1 < T; k += 2) {
      a.bd_kpanel = k;
      e = panel_launch(st, a, T - k - 1);
      if (e != cudaSuccess) return e;
      int nit = koff[k + 1] - koff[k];
      if (nit > 0) chol_update_tc_kernel<<<nit, U_THREADS, U_SMEM + 1024, st>>>(a, items + koff[k], 1, kug[k]);
      if (k + 2 < T) {
        KArgs b = a;
        b.bd_kpanel = k + 1;
        e = panel_launch(st, b, T - k - 2);
        if (e != cudaSuccess) return e;
        nit = koff[k + 2] - koff[k + 1];
        if (nit > 0) chol_update_tc_kernel<<<nit, U_THREADS, U_SMEM + 1024, st>>>(a, items + koff[k + 1], 2, kug[k + 1]);
      }
    }
  } else {
    for (int k = 0; k + 1 < T; ++k) {
      a.bd_kpanel = k;
      const int m = T - k - 1, np = m * (m + 1) / 2;
      e = panel_launch(st, a, m);
      if (e != cudaSuccess) return e;
      // quarter tiles while the whole ones would leave SMs idle
      if ((long long)np * a.nlane <= BD_SMS) chol_update_kernel<CT / 2><<<dim3(a.nlane, np, 4), 256, U64_SMEM, st>>>(a);
      else chol_update_kernel<CT><<<dim3(a.nlane, np), 256, U64_SMEM, st>>>(a);
    }
  }
  if (a.bd_refine) {
    e = cudaFuncSetAttribute(refine_residual_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, RT_SMEM);
    if (e != cudaSuccess) return e;
    const int TR = (3 * max_nmp + RT - 1) / RT;
    refine_residual_kernel<<<dim3(TR * (TR + 1) / 2, a.nlane), 256, RT_SMEM, st>>>(a);
    e = cudaFuncSetAttribute(refine_inverse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, RT_SMEM);
    if (e != cudaSuccess) return e;
    refine_inverse_kernel<<<dim3(TR, a.nlane), RT, RT_SMEM, st>>>(a);
  }
  return cudaGetLastError();
}

int bd_refactor_launches(int max_nmp, bool tc) {
  const int T = (3 * max_nmp + CT - 1) / CT;
  if (!tc) return 2 + 2 * (T - 1);
  int nl = 2;
  for (int k = 0; k + 1 < T; k += 2) nl += (k + 2 < T) ? 4 : 2;
  return nl;
}

// floats of the panel planes of a lane with N beads (tensor-core update)
long long bd_plane_floats(int nmp) {
  const int T = (3 * nmp + CT - 1) / CT;
  return 2LL * 2 * (T + 1) * PT;   // two panel slots of hi + lo planes
}

cudaError_t bd_step_launch(cudaStream_t st, const KArgs &a, int max_nmp) {
  bd_noise_kernel<<<dim3((max_nmp + 127) / 128, a.nlane), 128, 0, st>>>(a);
  if (a.bd_refine) {
    const size_t sm = (size_t)((3 * max_nmp + 1) & ~1) * sizeof(double) + (16 * RT + RT) * sizeof(double);
    cudaError_t e = cudaFuncSetAttribute(refine_trsv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    refine_trsv_kernel<<<a.nlane, TRSV_THREADS, sm, st>>>(a);
  }
  // four rows per warp once that still gives every SM two CTAs (64 rows): 32
  // chains of 100 to 1,000 beads 111 us against 187 with one row; below, the
  // rows of one warp would queue up behind one another on idle SMs
  if ((long long)3 * max_nmp * a.nlane >= 64LL * BD_SMS)
    bd_update_kernel<4><<<dim3((3 * max_nmp + 31) / 32, a.nlane), 256, 0, st>>>(a);
  else
    bd_update_kernel<1><<<dim3((3 * max_nmp + 7) / 8, a.nlane), 256, 0, st>>>(a);
  bd_force_kernel<<<dim3((max_nmp + 7) / 8, a.nlane), 256, 0, st>>>(a);
  return cudaGetLastError();
}

cudaError_t bd_force_launch(cudaStream_t st, const KArgs &a, int max_nmp) {
  bd_force_kernel<<<dim3((max_nmp + 7) / 8, a.nlane), 256, 0, st>>>(a);
  return cudaGetLastError();
}

} // namespace tis
