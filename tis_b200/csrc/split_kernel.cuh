// split_kernel.cuh -- one lane split over a cluster of 2 to 16 CTAs.
//
// A step of a lane is a short chain of dependent work: on one CTA a 1,199-bead
// lane keeps one of 148 SMs busy for 121 us a step, and what bounds it is that
// SM's issue rate and the latency of its longest items, not memory.  Split
// over 16 CTAs the same step takes 12.2 us; 599 beads in FP64 82 -> 9.5 us,
// 227 beads mixed 10.3 -> 5.8 us (8 CTAs), 65 beads FP64 11.2 -> 6.3 us (B200,
// event time of the step kernel).  Every mode of the lane kernel (KM_*) runs
// here, for both precisions, with or without a periodic box.
//
// Each CTA keeps the positions and pair parameters of every bead and owns a
// contiguous block of beads: their velocities and accelerations, excluded-
// volume rows and near lists, incidence slots and updates, and the bonded
// items whose first bead is one of them (divided by index instead, most of
// their results were remote stores of single values, and the barrier that
// waits for them took 9.3 k of a 400-nt step's 36 k cycles).  The charged
// rows of the electrostatic list are divided evenly, so an ion box (charges
// on every bead) is balanced too.  Results for another CTA's bead go there
// through distributed shared memory.
//
// One step is two phases between cluster barriers:
//   sweep   bonded terms, electrostatic rows, exv near lists, noise: warps
//           take chunks of items, longest kinds first, from a shared counter;
//           reads every position, writes slots and row sums.  The longest
//           serial chains are cut: a stack's two dihedrals run on two
//           threads, a hydrogen bond's three on four (14.3 k -> 5.3 k cycles
//           for one in FP64, with one reciprocal and corrections in place of five
//           divisions);
//   update  8 threads per own bead sum its slots (stored in incidence order,
//           so the reads are contiguous and need no index), add the row sums
//           and update v / a and x; then whole warps copy the block's new
//           positions to the other CTAs, 16 bytes a thread (stores of single
//           values cost ~2 cycles each on the SM-to-SM network), and only
//           the parts that the forces read (28 or 32 bytes a bead).
// Positions are not double buffered: nothing reads them in the update phase.
// A step whose lists must be rebuilt first does so from the old positions
// between its two halves, with one more barrier.
//
// Every bead's sums run in an order that depends on the lane's topology and
// lists only, so the results do not depend on the number of CTAs.
#pragma once
#include <cooperative_groups.h>
#include <cuda_pipeline.h>

#include <type_traits>

#include "lane_common.cuh"
#include "split_ewald.cuh"
#include "split_plan.cuh"

namespace tis {

namespace cg = cooperative_groups;

constexpr int MISC_ELIST = 14;   // flag: the partner lists of the charged rows are in shared memory


// the kernel's lambdas share its registers: outlined they would keep every captured value in local memory
#define SPLIT_INL __attribute__((always_inline))

// destination of a slot addressed by its number (rare paths): place
// slot_pos[k] of the lane's incidence lists, in the CTA that owns the bead
template <typename Real>
struct SplitDst {
  Real *slots;             // this CTA's copy
  const int *pos;          // slot_pos of the lane's topology
  const int *base;         // first incidence entry of each CTA
  unsigned magic;          // bead / own = mulhi(bead, magic)
};

template <typename Real>
__device__ __forceinline__ void put_slot(const SplitDst<Real> &d, size_t k, int bead, Real fx, Real fy, Real fz) {
  const int r = (int)__umulhi((unsigned)bead, d.magic);
  Real *p = cg::this_cluster().map_shared_rank(d.slots, r) + 3 * (ldro(d.pos + k) - d.base[r]);
  p[0] = fx; p[1] = fy; p[2] = fz;
}

// the same from a resolved destination word, CTA << 24 | place
template <typename Real>
__device__ __forceinline__ void put_word(Real *slots, int rank, uint32_t w, R3<Real> f) {
  const int r = (int)(w >> 24), k = 3 * (int)(w & 0xffffffu);
  if (r == rank) {
    slots[k] = f.x; slots[k + 1] = f.y; slots[k + 2] = f.z;
  } else {
    Real *p = cg::this_cluster().map_shared_rank(slots, r) + k;
    p[0] = f.x; p[1] = f.y; p[2] = f.z;
  }
}

// shared memory of a CTA: every bead's positions and pair parameters.  A4
// (with L3) is what a step sends and reads; the FP64 X and P of the other
// CTAs' beads are brought up to date only for a list build
template <typename Real>
struct SplitSmem {
  double *X, *Y, *Z, *PX, *PY, *PZ, *QX, *QY, *QZ;
  typename V4<Real>::T *A4;
  float *L3;               // mixed: pxyz - A4, so that A4 + L3 carries pxyz to ~2^-48
  Real *RE;                // exv radius, sqrt(eps)
  uint32_t *tcu;           // type | class << 4 | unit << 8 | cell << 16; cell: (X - P) / L of a periodic
                           // lane's bead, 5 bits a dimension, changed by list builds only
};

// FP64 coordinate of any bead during a sweep: the FP64 path's own copy; mixed,
// where a step sends FP32 hi and lo parts (2^-48), the owner's through
// distributed shared memory (nothing writes it between a step's barriers).
// For the terms that stay FP64 in both paths, few or rare
template <typename Real>
struct SplitCoord {
  const Real *A4;          // component of bead i at 4 i
  const double *X;         // the same component in its owner's copy
  unsigned magic;          // bead / own = mulhi(bead, magic)
  __device__ double operator[](int i) const {
    if constexpr (sizeof(Real) == 4) return cg::this_cluster().map_shared_rank(X, (int)__umulhi((unsigned)i, magic))[i];
    else return A4[4 * i];
  }
};
template <typename Real>
struct SplitView { SplitCoord<Real> PX, PY, PZ; };
template <typename Real>
__device__ __forceinline__ SplitView<Real> split_view(const SplitSmem<Real> &s, unsigned magic) {
  const Real *A = (const Real *)s.A4;
  return SplitView<Real>{{A, s.PX, magic}, {A + 1, s.PY, magic}, {A + 2, s.PZ, magic}};
}

template <typename Real>
__device__ __forceinline__ void split_pos(const SplitSmem<Real> &s, int i, double x, double y, double z) {
  const Real hx = (Real)x, hy = (Real)y, hz = (Real)z;
  s.A4[i].x = hx; s.A4[i].y = hy; s.A4[i].z = hz;
  if constexpr (sizeof(Real) == 4) {
    s.L3[3 * i] = (float)(x - (double)hx); s.L3[3 * i + 1] = (float)(y - (double)hy);
    s.L3[3 * i + 2] = (float)(z - (double)hz);
  }
}

// cells packed modulo 32; component d of the difference of two of them, -16
// .. 15 (beads of one bonded term that are further apart are not told apart
// from nearer ones)
__device__ __forceinline__ uint32_t cell_pack(double x, double y, double z) {
  return ((uint32_t)(int)x & 31u) | ((uint32_t)(int)y & 31u) << 5 | ((uint32_t)(int)z & 31u) << 10;
}
__device__ __forceinline__ int cell_diff(uint32_t p, uint32_t q, int d) {   // of two tcu words
  return (int)(((q >> (16 + 5 * d)) - (p >> (16 + 5 * d))) << 27) >> 27;
}

// image of the pair (i, j) fixed at the last rebuild, as x_j - x_i sees it
// (see mirror_shift): per dimension 0 none, 1 -L, 2 +L
template <typename S>
__device__ __forceinline__ int split_image(const KArgs &a, const S &s, int i, int j) {
  const double v[3] = {__dsub_rn(s.QX[j], s.QX[i]), __dsub_rn(s.QY[j], s.QY[i]), __dsub_rn(s.QZ[j], s.QZ[i])};
  int c = 0;
#pragma unroll
  for (int d = 2; d >= 0; --d) c = 3 * c + (v[d] > a.psizeh[d] ? 1 : (v[d] < -a.psizeh[d] ? 2 : 0));
  return c;
}
// place of set bit q of m (q < popc(m))
__device__ __forceinline__ int nth_bit(uint32_t m, int q) {
  int p = 0;
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const int c = __popc(m & ((1u << o) - 1u));
    if (q >= c) { q -= c; m >>= o; p += o; }
  }
  return p;
}

// b - a + k L (k in {-1, 0, 1}): across the box the two coordinates are ~L
// apart, so the rounding error of their difference is kept (TwoSum) and the
// box length taken in two parts; only the short result is rounded
__device__ __forceinline__ float diff_img(float a, float b, float k, double L) {
  const float s = b - a, bb = s - b, e = (b - (s - bb)) + (-a - bb);
  const float Lh = (float)L, Ll = (float)(L - (double)Lh);
  return fmaf(k, Lh, s) + fmaf(k, Ll, e);
}
__device__ __forceinline__ double diff_img(double a, double b, double k, double L) { return (b - a) + k * L; }

// One dihedral a-b-c-d of a stack or a hydrogen bond from u = x_a - x_b,
// w = x_c - x_b and z = x_c - x_d (up to a common sign): e = k d^2 with d
// the deviation from nat, and the derivative terms of the four beads, as
// force_dtrna_stack.F90:92-150 and force_dtrna_hbond15.F90:205-340 write
// them.  CAP: the hydrogen bonds' cap of nearly straight triples (maxc).
//
// Sums of products are written with their rounding (a b - c d = fma(a, b,
// -rn(c d)) and so on): left to the compiler, the variants of the kernel fuse
// one or the other product, and a lane's bits would depend on its number of
// CTAs.
__device__ __forceinline__ float mulr(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mulr(double a, double b) { return __dmul_rn(a, b); }
// a b + c d of the integration: FP64 as the reference evaluates it (see mad2)
template <typename Real> __device__ __forceinline__ double smad(double a, double b, double c, double d) {
  return sizeof(Real) == 8 ? __dadd_rn(__dmul_rn(a, b), __dmul_rn(c, d)) : fma(a, b, __dmul_rn(c, d));
}
template <typename Real> __device__ __forceinline__ Real det2(Real a, Real b, Real c, Real d) { return fma(a, b, -mulr(c, d)); }
template <typename Real> __device__ __forceinline__ Real sq3(Real x, Real y, Real z) { return fma(z, z, fma(y, y, mulr(x, x))); }
template <typename Real> __device__ __forceinline__ Real sdot(R3<Real> a, R3<Real> b) {
  return fma(a.z, b.z, fma(a.y, b.y, mulr(a.x, b.x)));
}
template <typename Real> __device__ __forceinline__ R3<Real> cross(R3<Real> a, R3<Real> b) {
  return R3<Real>{det2(a.y, b.z, a.z, b.y), det2(a.z, b.x, a.x, b.z), det2(a.x, b.y, a.y, b.x)};
}
// n / d from an inverse of d that is off by a few ulp
__device__ __forceinline__ double quot(double n, double d, double inv) {
  const double q = n * inv;
  return fma(fma(-q, d, n), inv, q);
}
// a vector's length and its inverse.  FP64: without the corrections by the
// residuals the length is off by 1.5 ulp, which the difference to the native
// length magnifies (forces of the chains 24 % further off than with sqrt)
__device__ __forceinline__ void length(float d2, float &d, float &r) { d = sqrtf(d2); r = __fdividef(1.0f, d); }
__device__ __forceinline__ void length(double d2, double &d, double &r) {
  r = rsqrt(d2);
  const double e = d2 * r;
  d = fma(fma(-e, e, d2), 0.5 * r, e);
  r = fma(fma(-d, r, 1.0), r, r);
}
template <typename Real> struct Dih { R3<Real> a, b, c, d; Real e; bool straight; };
template <typename Real, bool CAP>
__device__ __forceinline__ Dih<Real> dihedral(R3<Real> u, R3<Real> w, R3<Real> z, Real nat, Real k, Real maxc) {
  Dih<Real> o;
  const R3<Real> m = cross(u, w), n = cross(w, z);
  const Real w2 = sdot(w, w), uw = sdot(u, w), zw = sdot(z, w);
  Real m2 = sdot(m, m), n2 = sdot(n, n);
  if (CAP) {   // |cos| > maxc, compared as squares
    const Real uw2 = sdot(u, u) * w2, zw2 = sdot(z, z) * w2, mc2 = maxc * maxc;
    if (uw * uw > mc2 * uw2) m2 = uw2 * ((Real)1 - mc2);
    if (zw * zw > mc2 * zw2) n2 = zw2 * ((Real)1 - mc2);
    o.straight = false;
  } else {
    // mixed stacks: within ~2 degrees of straight FP32 is not enough (see term_stack)
    const Real lim = (Real)1e-3;
    o.straight = sizeof(Real) == 4 && (m2 < lim * sdot(u, u) * w2 || n2 < lim * w2 * sdot(z, z));
  }
  Real aw, ou, oz, im2, in2;   // |w|, uw / w2, zw / w2, 1 / m2, 1 / n2
  if constexpr (sizeof(Real) == 8) {
    // FP64 divisions are long dependent chains: one reciprocal square root
    // and one reciprocal stand for a square root and four divisions, each
    // result corrected by its residual to the rounding of the operation
    Real rw;
    length(w2, aw, rw);
    const Real iw2 = rw * rw, imn = (Real)1 / (m2 * n2);
    ou = quot(uw, w2, iw2); oz = quot(zw, w2, iw2);
    im2 = quot((Real)1, m2, n2 * imn); in2 = quot((Real)1, n2, m2 * imn);
  } else {
    aw = sqrt(w2); ou = fdiv(uw, w2); oz = fdiv(zw, w2); im2 = fdiv((Real)1, m2); in2 = fdiv((Real)1, n2);
  }
  const Real d = wrap_pi(atan2(sdot(u, n) * aw, sdot(m, n)) - nat);
  o.e = mulr(mulr(k, d), d);
  const Real pre = (Real)2 * k * d * aw, gi = pre * im2, gl = -pre * in2;
  o.a = R3<Real>{gi * m.x, gi * m.y, gi * m.z};
  o.d = R3<Real>{gl * n.x, gl * n.y, gl * n.z};
  const Real b1 = (Real)-1 + ou, c1 = (Real)-1 + oz;
  o.b = R3<Real>{det2(b1, o.a.x, oz, o.d.x), det2(b1, o.a.y, oz, o.d.y), det2(b1, o.a.z, oz, o.d.z)};
  o.c = R3<Real>{det2(c1, o.d.x, ou, o.a.x), det2(c1, o.d.y, ou, o.a.y), det2(c1, o.d.z, ou, o.a.z)};
  return o;
}
__device__ __forceinline__ float invsqrt(float x) { return rsqrtf(x); }
__device__ __forceinline__ double invsqrt(double x) { return rsqrt(x); }
template <typename Real> __device__ __forceinline__ R3<Real> add3(R3<Real> a, R3<Real> b) {
  return R3<Real>{a.x + b.x, a.y + b.y, a.z + b.z};
}
template <typename Real> __device__ __forceinline__ R3<Real> mul3(Real f, R3<Real> a) {
  return R3<Real>{f * a.x, f * a.y, f * a.z};
}
template <typename Real> __device__ __forceinline__ R3<Real> sel3(bool c, R3<Real> a, R3<Real> b) {
  return R3<Real>{c ? a.x : b.x, c ? a.y : b.y, c ? a.z : b.z};
}
template <typename Real> __device__ __forceinline__ R3<Real> shx3(R3<Real> a, int o) {
  return R3<Real>{__shfl_xor_sync(0xffffffffu, a.x, o), __shfl_xor_sync(0xffffffffu, a.y, o),
                  __shfl_xor_sync(0xffffffffu, a.z, o)};
}

// force_bangle.F90:103-147: the forces of one angle's beads (see term_angle)
template <typename Real>
__device__ __forceinline__ void split_angle(R3<Real> v21, R3<Real> v32, Real nat, Real cf, R3<Real> *f3) {
  const Real c11 = sdot(v21, v21), c22 = sdot(v32, v32), c21 = sdot(v32, v21), rs = invsqrt(c11 * c22);
  Real co = -c21 * rs;
  if (co > (Real)1) co = 1; else if (co < (Real)-1) co = -1;
  Real th, t3;
  if (sizeof(Real) == 4 && fabs(co) > (Real)0.99) {
    const R3<Real> cr = cross(v21, v32);
    t3 = sdot(cr, cr);
    th = atan2(sqrt(t3), -c21);
  } else {
    th = acos(co);
    t3 = det2(c11, c22, c21, c21);
  }
  if (t3 <= (Real)1) t3 = 1;
  const Real f = cf < (Real)1.0e-6 ? (Real)0 : (Real)2 * cf * (th - nat) * invsqrt(t3);
  Real a1, a2;
  if constexpr (sizeof(Real) == 8) { const Real r2 = rs * rs; a1 = quot(c21, c11, c22 * r2); a2 = quot(c21, c22, c11 * r2); }
  else { a1 = fdiv(c21, c11); a2 = fdiv(c21, c22); }
  const R3<Real> A{fma(v21.x, a1, -v32.x), fma(v21.y, a1, -v32.y), fma(v21.z, a1, -v32.z)};
  const R3<Real> B{fma(v32.x, a2, -v21.x), fma(v32.y, a2, -v21.y), fma(v32.z, a2, -v21.z)};
  f3[0] = mul3(-f, A);
  f3[1] = mul3(f, R3<Real>{A.x - B.x, A.y - B.y, A.z - B.z});
  f3[2] = mul3(f, B);
}

// asynchronous copies global -> shared, all in flight together
__device__ __forceinline__ void acopy16(void *dst, const void *src) { __pipeline_memcpy_async(dst, src, 16); }
__device__ __forceinline__ void acopy8(void *dst, const void *src) { __pipeline_memcpy_async(dst, src, 8); }
__device__ __forceinline__ void acopy4(void *dst, const void *src) { __pipeline_memcpy_async(dst, src, 4); }

template <typename Real, int NT, bool PER>
__global__ void __launch_bounds__(NT) split_kernel(const __grid_constant__ KArgs a) {
  typedef typename V4<Real>::T V;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if constexpr (PER)
    if (a.ew_nwork && threadIdx.x == 0) ew_signal(a, EWS_ARRIVED);
  if constexpr (PER)
    if (a.ew_nwork && blockIdx.x >= gridDim.x - (unsigned)a.ew_nwork) {
      ewald_worker<NT>(a, smem_raw);
      return;
    }
  const cg::cluster_group cl = cg::this_cluster();
  const int nr = a.nsplit, rank = (int)cl.block_rank();
  const int lane = (a.only_lane >= 0) ? a.only_lane
                                      : (a.lane_order ? a.lane_order[blockIdx.x / nr] : (int)(blockIdx.x / nr));
  if (lane >= a.nlane) return;
  // replicas that have reached their exchange step wait (time_integral.F90:134)
  if (a.lane_nsteps && (a.mode == KM_XSTEP || a.mode == KM_VSTEP || a.mode == KM_VXSTEP) &&
      a.step_k >= a.lane_nsteps[lane])
    return;
  const int lane_steps = (a.lane_nsteps && a.mode == KM_STEP) ? min(a.nsteps, a.lane_nsteps[lane]) : a.nsteps;
  if (a.mode == KM_STEP && lane_steps <= 0) return;
  const LaneDesc L = a.lanes[lane];
  const TopDesc T = a.tops[L.top];
  const int N = T.nmp, NQ = (a.i_ele != 0) ? T.nq : 0, W = (N + 31) >> 5, nu = T.nunit;
  const int tid = threadIdx.x, warp = tid >> 5, lid = tid & 31;
  constexpr int NW = NT / 32;
  const bool skin = a.n_step_neighbor <= 0;
  LaneState &st = a.lstate[lane];
  const SplitPlan &pl = a.sp;
  SplitSmem<Real> s;
  unsigned char *sm = smem_raw;
  const int np = pl.np, OS = pl.own;      // component strides of the positions and of the own beads
  const int own = split_own(N, nr), rows = (NQ + nr - 1) / nr;
  s.X = (double *)(sm + pl.X); s.Y = s.X + np; s.Z = s.Y + np;
  s.PX = (double *)(sm + pl.P); s.PY = s.PX + np; s.PZ = s.PY + np;
  s.QX = (double *)(sm + pl.Q); s.QY = s.QX + np; s.QZ = s.QY + np;
  s.A4 = (V *)(sm + pl.A4);
  s.L3 = (float *)(sm + pl.L3);
  s.RE = (Real *)(sm + pl.RE);
  s.tcu = (uint32_t *)(sm + pl.tcu);
  auto typ = [&](int i) SPLIT_INL { return (int)(s.tcu[i] & 15u); };
  auto cls = [&](int i) SPLIT_INL { return (int)(s.tcu[i] >> 4 & 15u); };
  auto unit = [&](int i) SPLIT_INL { return (int)(s.tcu[i] >> 8 & 255u); };
  const int lo = min(N, rank * own), hi = min(N, lo + own), nown = hi - lo;
  double *Vv = (double *)(sm + pl.V), *Av = Vv + 3 * OS, *Dv = Av + 3 * OS;   // component d of own bead li at d OS + li
  double *DD = (double *)(sm + pl.DD), *C1 = (double *)(sm + pl.C1);
  const double *C2 = (double *)(sm + pl.C), *C3 = C2 + OS, *C4 = C3 + OS, *RC = C4 + OS;
  double *NZ = (double *)(sm + pl.NZ), *exF = (double *)(sm + pl.exF), *dhF = (double *)(sm + pl.dhF);
  const Real *scr = (Real *)(sm + pl.scr);
  float4 *NR4 = (float4 *)(sm + pl.NR4);
  uint16_t *near = (uint16_t *)(sm + pl.near);
  uint8_t *ncnt = (uint8_t *)(sm + pl.ncnt);
  uint32_t *mexv = (uint32_t *)(sm + pl.mexv), *mele = (uint32_t *)(sm + pl.mele);
  Real *slots = (Real *)(sm + pl.slots);
  const int *iptr = (int *)(sm + pl.iptr), *base = (int *)(sm + pl.base), *qb = (int *)(sm + pl.qb);
  int *exc = (int *)(sm + pl.exc);
  uint8_t *hbf = (uint8_t *)(sm + pl.hbf);
  const double *rn2 = (double *)(sm + pl.rn2);
  double *red = (double *)(sm + pl.red), *redc = red + 64;
  // [parity][CTA], float bits: largest dot_product(dxyz, dxyz), rounded up; largest squared displacement
  // since the near lists were recorded
  int2 *dmax = (int2 *)(redc + 2 * SPLIT_MAX);
  float4 *imgf = (float4 *)(sm + pl.img);
  double4 *imgd = (double4 *)(sm + pl.img);
  int *misc = (int *)(sm + pl.misc);
  uint16_t *elist = (uint16_t *)(sm + pl.elist);
  int *eoff = (int *)(sm + pl.eoff);       // first entry of each charged row's list
  const double *u0s = (double *)(sm + pl.u0);
  const unsigned magic = (unsigned)((0x100000000ull + (unsigned)own - 1) / (unsigned)own);   // exact for beads < 2^16
  const SplitDst<Real> dst{slots, a.slot_pos + T.sp0, base, magic};
  // this CTA's share of the charged rows and of each kind of bonded item
  const int kq_lo = min(NQ, rank * rows), nrow = min(NQ, kq_lo + rows) - kq_lo;
  const unsigned char *comm = a.split_blob + T.sp_blob, *mine = comm + (size_t)rank * (pl.stat - pl.comm);
  const int *cnt = (const int *)(mine + pl.cnt);   // bonded items of this CTA
  const int nh = ldro(cnt), nst = ldro(cnt + 1), nts = ldro(cnt + 2), nba = ldro(cnt + 3), nbd = ldro(cnt + 4);
  const int *hbk = (const int *)(sm + pl.hbk), *stk = (const int *)(sm + pl.stk), *tsk = (const int *)(sm + pl.tsk);
  const int label = st.label;
  const long long istep0 = st.istep;   // written by CTA 0 after the last cluster barrier

  // ---- load: every copy is asynchronous, so the arrays' latencies overlap
  const bool lists_new = a.mode == KM_NEIGHBOR || a.mode == KM_PRE;
  {
    for (unsigned q = 16 * tid; q < pl.stat; q += 16 * NT) acopy16(sm + q, (q < pl.comm ? comm : mine) + q);
    const size_t o = 3 * (size_t)L.state0;
    for (int q = tid; q < 3 * N; q += NT) {
      const int i = q / 3, k = (q - 3 * i) * np + i;
      acopy8(s.X + k, a.xyz + o + q);
      if (PER) { acopy8(s.PX + k, a.pxyz + o + q); acopy8(s.QX + k, a.p0xyz + o + q); }
    }
    for (int q = tid; q < 3 * nown; q += NT) {
      const int li = q / 3, k = (q - 3 * li) * OS + li;
      const size_t g = o + 3 * (size_t)lo + q;
      acopy8(Vv + k, a.velo + g); acopy8(Av + k, a.accel + g);
      if (skin) acopy8(Dv + k, a.dxyz + g);
    }
    const double *c1 = a.lab_c1 + a.lab_c1off[label] + lo, *u0 = a.lab_u0 + a.lab_u0off[label];
    for (int li = tid; li < nown; li += NT) acopy8(C1 + li, c1 + li);
    for (int k = tid; k < nst; k += NT) acopy8((double *)u0s + k, u0 + ldro((const int *)(mine + pl.stk) + k));
    if (!lists_new) {
      const uint32_t *gm = a.mask + L.mask0;
      for (int k = tid; k < nown * W; k += NT) acopy4(mexv + k, gm + (size_t)lo * W + k);
      for (int k = warp; k < nrow; k += NW) {
        const uint32_t *row = gm + (size_t)N * W + (size_t)ldro(a.q_bead + T.q0 + kq_lo + k) * W;
        for (int w = lid; w < W; w += 32) acopy4(mele + k * W + w, row + w);
      }
    }
    __pipeline_commit();
    for (int k = tid; k < 3 * T.sp_ninc; k += NT) slots[k] = (Real)0;
    for (int k = tid; k < 3 * OS; k += NT) dhF[k] = 0.0;
    for (int k = tid; k < T.nsite; k += NT) exc[k] = 0;
    for (int k = tid; k < nh; k += NT) hbf[k] = a.hb_flag[L.hb0 + ldro((const int *)(mine + pl.hbk) + k)];
    if (tid < SPLIT_MISC) misc[tid] = tid == MISC_NEAR_BAD ? 1 : (tid == MISC_CHUNK ? NW : 0);
    if (tid < 2 * SPLIT_MAX) dmax[tid] = make_int2(0, 0);
    if (PER && tid < 27) {   // the shift of each image as multiples of the box
      const int c[3] = {tid % 3, (tid / 3) % 3, tid / 9};
      auto k = [](int q) { return q == 0 ? 0.0 : (q == 1 ? -1.0 : 1.0); };
      if (sizeof(Real) == 4) imgf[tid] = make_float4((float)k(c[0]), (float)k(c[1]), (float)k(c[2]), 0.f);
      else imgd[tid] = make_double4(k(c[0]), k(c[1]), k(c[2]), 0.0);
    }
    for (int i = tid; i < N; i += NT) s.A4[i].w = (Real)bead_charge(a, label, T.bead0 + i);
    if (tid == 0) { V far; far.x = far.y = far.z = (Real)1.0e6; far.w = 0; s.A4[np] = far; }
    __pipeline_wait_prior(0);
    __syncthreads();
    for (int i = tid; i < N; i += NT) {
      split_pos<Real>(s, i, s.PX[i], s.PY[i], s.PZ[i]);
      if (PER) s.tcu[i] |= cell_pack(rint((s.X[i] - s.PX[i]) / a.psize[0]), rint((s.Y[i] - s.PY[i]) / a.psize[1]),
                                     rint((s.Z[i] - s.PZ[i]) / a.psize[2])) << 16;
    }
  }
  cl.sync();   // loaded; and every CTA runs before any distributed access

  // x_j - x_i of the pair (i, j) with its image
  auto pair_diff = [&](const V &pi, const V &pj, int img, Real &x, Real &y, Real &z) SPLIT_INL {
    if constexpr (PER) {
      Real kx, ky, kz;
      if constexpr (sizeof(Real) == 4) { const float4 k = imgf[img]; kx = k.x; ky = k.y; kz = k.z; }
      else { const double4 k = imgd[img]; kx = k.x; ky = k.y; kz = k.z; }
      x = diff_img(pi.x, pj.x, kx, a.psize[0]); y = diff_img(pi.y, pj.y, ky, a.psize[1]);
      z = diff_img(pi.z, pj.z, kz, a.psize[2]);
    } else {
      x = pj.x - pi.x; y = pj.y - pi.y; z = pj.z - pi.z;
    }
  };

  const bool ewald = a.i_ele == 2, coul = a.i_ele == 3;
  const int LQ = split_row_lanes(NQ, ewald), RW = 32 / LQ;
  // x_j - x_i of the bonded terms in W, in FP32 from the hi and lo parts,
  // rounded once (FP64 terms of the mixed path: from the FP64 positions).  Periodic: of the unwrapped positions (bonds, angles,
  // stacks), i.e. of the wrapped ones and the beads' cells, or the nearest
  // image (hydrogen bonds).  Across the box the two coordinates are ~L apart,
  // so the rounding error of their difference is kept (TwoSum)
  auto bvec = [&](auto nearest, auto w, int i, int j) SPLIT_INL {
    typedef decltype(w) Wt;
    constexpr bool NEAREST = decltype(nearest)::value;
    const V p = s.A4[i], q = s.A4[j];
    uint32_t ci = 0, cj = 0;
    if (PER && !NEAREST) { ci = s.tcu[i]; cj = s.tcu[j]; }
    if constexpr (sizeof(Wt) == 4) {
      const float *l = s.L3 + 3 * i, *m = s.L3 + 3 * j;
      auto d1 = [&](float x, float y, float lx, float ly, int d) SPLIT_INL {
        const float t = y - x, bb = t - y, e = (y - (t - bb)) + (-x - bb) + (ly - lx);
        if (!PER) return t + e;
        float k;
        if (NEAREST) { const float h = (float)a.psizeh[d]; k = t > h ? -1.0f : (t < -h ? 1.0f : 0.0f); }
        else k = (float)cell_diff(ci, cj, d);
        const float Lh = (float)a.psize[d], Ll = (float)(a.psize[d] - (double)Lh);
        return fmaf(k, Lh, t) + fmaf(k, Ll, e);
      };
      return R3<Wt>{d1(p.x, q.x, l[0], m[0], 0), d1(p.y, q.y, l[1], m[1], 1), d1(p.z, q.z, l[2], m[2], 2)};
    } else {
      if constexpr (sizeof(Real) == 4) {   // the owners' unwrapped FP64 positions (see SplitCoord)
        static_assert(!NEAREST, "");
        const double *xi = cl.map_shared_rank(s.X, (int)__umulhi((unsigned)i, magic)) + i;
        const double *xj = cl.map_shared_rank(s.X, (int)__umulhi((unsigned)j, magic)) + j;
        return R3<Wt>{xj[0] - xi[0], xj[np] - xi[np], xj[2 * np] - xi[2 * np]};
      }
      const double px = (double)p.x, py = (double)p.y, pz = (double)p.z;
      const double qx = (double)q.x, qy = (double)q.y, qz = (double)q.z;
      if (PER && !NEAREST) {
        auto d1 = [&](double x, double y, int d) SPLIT_INL {
          const double t = y - x, bb = t - y, e = (y - (t - bb)) + (-x - bb);
          return fma((double)cell_diff(ci, cj, d), a.psize[d], t) + e;
        };
        return R3<Wt>{d1(px, qx, 0), d1(py, qy, 1), d1(pz, qz, 2)};
      }
      double x = qx - px, y = qy - py, z = qz - pz;
      if (PER) { pb1(x, a.psize[0], a.psizeh[0]); pb1(y, a.psize[1], a.psizeh[1]); pb1(z, a.psize[2], a.psizeh[2]); }
      return R3<Wt>{x, y, z};
    }
  };
  auto rvec = [&](auto w, int i, int j) SPLIT_INL { return bvec(std::false_type(), w, i, j); };
  // partner lists of the charged rows from their bit rows (with the image of
  // each pair when periodic): lane l expands words l, l + 32, ...
  // (called by the whole CTA; misc[MISC_ELIST]: they fit)
  auto expand_rows = [&]() SPLIT_INL {
    for (int k = warp; k < nrow; k += NW) {
      int n = 0;
      for (int w = lid; w < W; w += 32) n += __popc(mele[k * W + w]);
      n = __reduce_add_sync(0xffffffffu, n);
      if (lid == 0) eoff[k + 1] = (n + 2 * LQ - 1) / (2 * LQ) * (2 * LQ);   // whole rounds of the row's threads
    }
    __syncthreads();
    if (warp == 0) {
      int sum = 0;
      for (int k0 = 0; k0 < nrow; k0 += 32) {
        int v = k0 + lid < nrow ? eoff[k0 + lid + 1] : 0;
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(0xffffffffu, v, o);
          if (lid >= o) v += t;
        }
        if (k0 + lid < nrow) eoff[k0 + lid + 1] = sum + v;
        sum += __shfl_sync(0xffffffffu, v, 31);
      }
      if (lid == 0) { eoff[0] = 0; misc[MISC_ELIST] = sum <= (int)pl.ecap; }
    }
    __syncthreads();
    if (!misc[MISC_ELIST]) return;
    for (int k = warp; k < nrow; k += NW) {
      const int i = qb[kq_lo + k], end = eoff[k + 1] - eoff[k];
      uint16_t *out = elist + eoff[k];
      int n = 0;
      for (int w0 = 0; w0 < W; w0 += 32) {
        uint32_t m = (w0 + lid < W) ? mele[k * W + w0 + lid] : 0u;
        int incl = __popc(m);
        const int c = incl;
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(0xffffffffu, incl, o);
          if (lid >= o) incl += t;
        }
        int at = n + incl - c;
        n += __shfl_sync(0xffffffffu, incl, 31);
        while (m) {
          const int j = ((w0 + lid) << 5) + __ffs(m) - 1;
          m &= m - 1;
          out[at++] = (uint16_t)(PER ? (j | (split_image(a, s, i, j) << SP_IMG)) : j);
        }
      }
      // padded with the far bead
      if (n + lid < end) out[n + lid] = (uint16_t)np;
      if (n + 32 + lid < end) out[n + 32 + lid] = (uint16_t)np;
    }
  };

  // ---- list build (see lane_kernel.cu build_lists for the rules): a warp
  // tests one own row, lane l bead 32 w + l, and writes its words by ballot;
  // mixed precision screens in FP32 and takes the FP64 test of the reference
  // only within the rounding of the screen
  auto build = [&](long long is, bool loaded) SPLIT_INL {
    if (!loaded) {
      // the FP64 positions of the other CTAs' beads (nobody moves beads now)
      bool units = false;   // the unit prescreen sums unwrapped positions
      if (PER)
        for (int u = 0, n = 0; u < nu; ++u) { n += a.u_class[T.unit0 + u] != 4; units = n > 1; }
      for (int i = tid; i < N; i += NT) {
        const int r = (int)__umulhi((unsigned)i, magic);
        if (r == rank) continue;
        const double *P = cl.map_shared_rank(s.PX, r);
        s.PX[i] = P[i]; s.PY[i] = P[np + i]; s.PZ[i] = P[2 * np + i];
        if (PER && units) {
          const double *X = cl.map_shared_rank(s.X, r);
          s.X[i] = X[i]; s.Y[i] = X[np + i]; s.Z[i] = X[2 * np + i];
        }
      }
      cl.sync();   // (the owners wrap theirs below)
    }
    if (PER) {
      for (int i = tid; i < N; i += NT) {
        const double x = wrap1(s.PX[i], a.psize[0]), y = wrap1(s.PY[i], a.psize[1]), z = wrap1(s.PZ[i], a.psize[2]);
        const uint32_t moved = cell_pack(rint((s.PX[i] - x) / a.psize[0]), rint((s.PY[i] - y) / a.psize[1]),
                                         rint((s.PZ[i] - z) / a.psize[2]));
        if (moved) {
          const uint32_t t = s.tcu[i], c = t >> 16;
          s.tcu[i] = (t & 0xffffu) | ((c + (moved & 31u)) & 31u) << 16 | (((c >> 5) + (moved >> 5)) & 31u) << 21 |
                     (((c >> 10) + (moved >> 10)) & 31u) << 26;
        }
        s.PX[i] = x; s.PY[i] = y; s.PZ[i] = z;
        s.QX[i] = x; s.QY[i] = y; s.QZ[i] = z;
        split_pos<Real>(s, i, x, y, z);
      }
    }
    // coordinates beyond 2048 A (or not finite) switch the screen off
    int far_l = 0;
    if (sizeof(Real) == 4)
      for (int i = tid; i < N; i += NT)
        far_l |= !(fabs(s.PX[i]) < 2048.0 && fabs(s.PY[i]) < 2048.0 && fabs(s.PZ[i]) < 2048.0);
    int *unit_ok = misc + SPLIT_MISC;
    if (tid == 0) {
      misc[MISC_NEXV] = 0; misc[MISC_NELE] = 0; misc[MISC_NEAR_BAD] = 1;
      // unit prescreen (neighbor_pre.F90:174-252)
      double cm[3 * 32], md[32];
      if (nu > 1)
        for (int u = 0; u < nu && u < 32; ++u) {
          const int is_ = a.u_lunit[2 * (T.unit0 + u)], ie = a.u_lunit[2 * (T.unit0 + u) + 1];
          md[u] = 0; cm[3 * u] = cm[3 * u + 1] = cm[3 * u + 2] = 0;
          bool need = false;   // only a pair of two different units that are no ions is tested
          if (a.u_class[T.unit0 + u] != 4)
            for (int v = 0; v < nu; ++v) need |= v != u && a.u_class[T.unit0 + v] != 4;
          if (!need) continue;
          double sx = 0, sy = 0, sz = 0;
          for (int i = is_; i <= ie; ++i) { sx += s.X[i]; sy += s.Y[i]; sz += s.Z[i]; }
          const double n = (double)(ie - is_ + 1);
          cm[3 * u] = sx / n; cm[3 * u + 1] = sy / n; cm[3 * u + 2] = sz / n;
          double m = 0;
          for (int i = is_; i <= ie; ++i) {
            const double dx = s.X[i] - cm[3 * u], dy = s.Y[i] - cm[3 * u + 1], dz = s.Z[i] - cm[3 * u + 2];
            const double d2 = dx * dx + dy * dy + dz * dz;
            if (d2 > m) m = d2;
          }
          md[u] = sqrt(m);
          if (PER) for (int d = 0; d < 3; ++d) cm[3 * u + d] = wrap1(cm[3 * u + d], a.psize[d]);
        }
      for (int u = 0; u < nu; ++u)
        for (int v = u; v < nu; ++v) {
          int ok = 1;
          if (!(a.u_class[T.unit0 + u] == 4 || a.u_class[T.unit0 + v] == 4 || u == v || u >= 32 || v >= 32)) {
            double w[3] = {cm[3 * v] - cm[3 * u], cm[3 * v + 1] - cm[3 * u + 1], cm[3 * v + 2] - cm[3 * u + 2]};
            if (PER) for (int d = 0; d < 3; ++d) pb1(w[d], a.psize[d], a.psizeh[d]);
            ok = sqrt(w[0] * w[0] + w[1] * w[1] + w[2] * w[2]) < md[u] + md[v] + sqrt(rn2[u * nu + v]);
          }
          unit_ok[u * nu + v] = ok;
          unit_ok[v * nu + u] = ok;
        }
    }
    const bool exact_only = __syncthreads_or(far_l) != 0 || sizeof(Real) == 8;
    const double rele2 = (a.i_ele != 0) ? a.lab_rele2[label] : -1.0;
    uint8_t *mir = PER ? (a.mirror + L.mirror0) : nullptr;
    uint32_t *gm = a.mask + L.mask0;
    // the distance test of (i, j) against rc2; im receives the mirror index when inside and periodic
    auto inside = [&](int i, int j, double rc2, int &im) SPLIT_INL {
      if (!exact_only) {
        const V pi = s.A4[i], pj = s.A4[j];
        float x = (float)(pj.x - pi.x), y = (float)(pj.y - pi.y), z = (float)(pj.z - pi.z);
        if (PER) {
          const float hx = (float)a.psizeh[0], hy = (float)a.psizeh[1], hz = (float)a.psizeh[2];
          x = fminf(fabsf(x), fabsf(fabsf(x) - 2.0f * hx)); y = fminf(fabsf(y), fabsf(fabsf(y) - 2.0f * hy));
          z = fminf(fabsf(z), fabsf(fabsf(z) - 2.0f * hz));
        }
        const float d2 = x * x + y * y + z * z, rc = (float)rc2;
        // |error of d2| < 2 d (coordinate rounding 4.3e-4 at 2048 A) + 1e-6 d2, d near the cutoff
        const float band = rc * 2.0e-3f + 0.02f;
        if (d2 > rc + band) return false;
        if (!PER && d2 < rc - band) return true;
      }
      double v0 = __dsub_rn(s.PX[j], s.PX[i]), v1 = __dsub_rn(s.PY[j], s.PY[i]), v2 = __dsub_rn(s.PZ[j], s.PZ[i]);
      if (PER) {
        const int m0 = pb1(v0, a.psize[0], a.psizeh[0]);
        const int m1 = pb1(v1, a.psize[1], a.psizeh[1]);
        const int m2 = pb1(v2, a.psize[2], a.psizeh[2]);
        im = 9 * m0 + 3 * m1 + m2 + 1;
      }
      return __dadd_rn(__dadd_rn(sqr_rn(v0), sqr_rn(v1)), sqr_rn(v2)) < rc2;
    };
    int nexv = 0, nele = 0;   // lane 0 of each warp
    for (int li = warp; li < nown; li += NW) {
      const int i = lo + li, ui = unit(i), ci = cls(i), ti = typ(i);
      const int nsep_i = (ti == 2) ? a.nsep[0] : (ti == 4 ? a.nsep[1] : (ti == 3 ? a.nsep[2] : -1));
      const bool qi = fabs((double)s.A4[i].w) > 1.0e-6;
      for (int w = 0; w < W; ++w) {
        const int j = (w << 5) + lid;
        bool ex = false;
        if (j < N && j != i) {
          const int uj = unit(j), cj = cls(j);
          ex = true;
          if (ui == uj) {
            if (ci == 2 /* RNA */) {   // the lower bead's separation (neighbor_assign.F90:481-557)
              const int tl = j > i ? ti : typ(j);
              const int ns = j > i ? nsep_i : ((tl == 2) ? a.nsep[0] : (tl == 4 ? a.nsep[1] : (tl == 3 ? a.nsep[2] : -1)));
              if (abs(j - i) < ns) ex = false;
            }
          } else if (!unit_ok[ui * nu + uj] ||
                     !((ci == 2 && cj == 2) || (ci == 2 && cj == 4) || (ci == 4 && cj == 2) ||
                       (ci == 4 && cj == 3) || (ci == 3 && cj == 4))) {
            ex = false;
          } else if (a.dt19 && ((ci == 2 && cj == 4) || (ci == 4 && cj == 2))) {
            // neighbor_assign.F90:524-537: no exv between a charged phosphate and an ion (the lower bead first)
            const int l2 = min(i, j), h2 = max(i, j);
            const int pb = (typ(l2) == 2) ? l2 : ((typ(h2) == 2) ? h2 : -1);
            if (pb >= 0 && (pb == i ? qi : fabs((double)s.A4[pb].w) > 1.0e-6)) ex = false;
          }
          if (ex) {
            int im = 27;
            // the pair test takes the lower bead first (its rounding is even in the order)
            ex = inside(min(i, j), max(i, j), rn2[ui * nu + uj], im);
            if (ex && mir && j > i) mir[(size_t)i * N + j] = (uint8_t)im;
          }
        }
        const uint32_t m = __ballot_sync(0xffffffffu, ex);
        if (lid == 0) {
          mexv[li * W + w] = m;
          gm[(size_t)i * W + w] = m;
          const int b = i - (w << 5);   // bits j > i
          nexv += __popc(b < 0 ? m : (b >= 31 ? 0u : m & ~((2u << b) - 1u)));
        }
      }
    }
    for (int k = warp; k < nrow; k += NW) {
      const int i = qb[kq_lo + k], ui = unit(i);
      const bool qi = fabs((double)s.A4[i].w) >= 1.0e-6;
      for (int w = 0; w < W; ++w) {
        const int j = (w << 5) + lid;
        bool el = false;
        if (qi && j < N && j != i && fabs((double)s.A4[j].w) >= 1.0e-6 && unit_ok[ui * nu + unit(j)]) {
          int im = 27;
          el = inside(min(i, j), max(i, j), rele2, im);
          if (el && mir && j > i) mir[(size_t)i * N + j] = (uint8_t)im;
        }
        const uint32_t m = __ballot_sync(0xffffffffu, el);
        if (lid == 0) {
          mele[k * W + w] = m;
          gm[(size_t)N * W + (size_t)i * W + w] = m;
          const int b = i - (w << 5);
          nele += __popc(b < 0 ? m : (b >= 31 ? 0u : m & ~((2u << b) - 1u)));
        }
      }
    }
    if (nexv) atomicAdd(&misc[MISC_NEXV], nexv);
    if (nele) atomicAdd(&misc[MISC_NELE], nele);
    // hbond neighbour flags (neighbor_list_hb.F90:335-354)
    for (int k = tid; k < nh; k += NT) {
      const int h = hbk[k], *m = a.hb_idx + 6 * (size_t)(T.hb0 + h);
      const int m0 = ldro(m), m1 = ldro(m + 1);
      double v0 = __dsub_rn(s.PX[m0], s.PX[m1]), v1 = __dsub_rn(s.PY[m0], s.PY[m1]), v2 = __dsub_rn(s.PZ[m0], s.PZ[m1]);
      if (PER) { pb1(v0, a.psize[0], a.psizeh[0]); pb1(v1, a.psize[1], a.psizeh[1]); pb1(v2, a.psize[2], a.psizeh[2]); }
      const int on = __dadd_rn(__dadd_rn(sqr_rn(v0), sqr_rn(v1)), sqr_rn(v2)) < a.hb_nd2[T.hb0 + h] ? 1 : 0;
      hbf[k] = (uint8_t)((hbf[k] & 2) | on);   // bit 1: the slots hold a force
      a.hb_flag[L.hb0 + h] = (uint8_t)on;
    }
    __syncthreads();
    expand_rows();
    // every CTA has finished with the positions and counts
    cl.sync();
    if (tid == 0 && rank == 0) {
      int ne = 0, nl = 0;
      for (int r = 0; r < nr; ++r) {
        const int *m = cl.map_shared_rank(misc, r);
        ne += m[MISC_NEXV]; nl += m[MISC_NELE];
      }
      rebuild_counts(st, ne, nl, is);
    }
  };

  // ---- skin trigger, exact: the top two d2 of every CTA's beads; called by
  // every thread of every CTA
  auto skin_exact = [&](bool from_dxyz) SPLIT_INL {
    double m1 = 0.0, m2 = 0.0;
    for (int li = tid; li < nown; li += NT)
      top2_add(m1, m2, from_dxyz ? disp2(Dv[li], Dv[OS + li], Dv[2 * OS + li]) : DD[li]);
    top2_store(m1, m2, red);
    __syncthreads();
    if (warp == 0) {
      m1 = lid < NW ? red[2 * lid] : 0.0; m2 = lid < NW ? red[2 * lid + 1] : 0.0;
      top2_warp(m1, m2);
      if (lid < nr) {
        double *o = cl.map_shared_rank(redc, lid);
        o[2 * rank] = m1; o[2 * rank + 1] = m2;
      }
    }
    cl.sync();
    m1 = lid < nr ? redc[2 * lid] : 0.0; m2 = lid < nr ? redc[2 * lid + 1] : 0.0;
    return skin_decide(m1, m2, a.neigh_margin);
  };

  // ---- x update (time_integral.F90:152-161) of own bead li, called by whole
  // warps (group of SG threads per bead, components on threads 0..2): into
  // this CTA's copy; send() then hands the block to the other CTAs
  const int g = tid & (SG - 1), grp = tid / SG;
  constexpr int NG = NT / SG;
  auto xmove = [&](int li, bool valid, bool fire) SPLIT_INL {
    const int i = lo + li;
    if (valid && g < 3) {
      const int q = g * OS + li;
      const double dx = smad<Real>(C4[li], Vv[q], a.tstep2, Av[q]);
      const double nx = s.X[g * np + i] + dx;
      s.X[g * np + i] = nx;
      double p = nx;
      if (PER) { p = s.PX[g * np + i] + dx; s.PX[g * np + i] = p; }
      if (skin) Dv[q] = fire ? dx : Dv[q] + dx;   // dxyz restarts at a rebuild (time_integral.F90:89)
      const Real h = (Real)p;
      (&s.A4[i].x)[g] = h;
      if constexpr (sizeof(Real) == 4) s.L3[3 * i + g] = (float)(p - (double)h);
    }
    __syncwarp();
    int bits = 0, nbits = 0;   // float bits, order-preserving for values >= 0
    if (valid && g == 0) {
      const V p = s.A4[i];
      const float4 r = NR4[li];
      const float ex = (float)p.x - r.x, ey = (float)p.y - r.y, ez = (float)p.z - r.z, e2 = sq3(ex, ey, ez);
      nbits = e2 >= 0.0f ? __float_as_int(e2) : 0x7f000000;   // (before the first recording NR4 holds anything)
      if (skin) {
        const double d2 = disp2(Dv[li], Dv[OS + li], Dv[2 * OS + li]);
        DD[li] = d2;
        bits = __float_as_int(__double2float_ru(d2));
      }
    }
    nbits = __reduce_max_sync(0xffffffffu, nbits);
    if (lid == 0) atomicMax(&misc[MISC_NEAR_DISP], nbits);
    if (skin) {
      bits = __reduce_max_sync(0xffffffffu, bits);
      if (lid == 0) atomicMax(&misc[MISC_DMAX], bits);
    }
  };
  // the block's new positions (and displacement maximum) to every other CTA,
  // 16 bytes per thread, whole warps per CTA: scattered stores of single
  // values cost ~2 cycles each on the SM-to-SM network
  auto send = [&](int par) SPLIT_INL {
    __syncthreads();
    constexpr int PV = sizeof(V) / 16;
    const int avail = max(((N + 3) & ~3) - lo, 0);   // beads from lo on: the last block is shorter
    const int nA = min(own, avail) * PV, nL = sizeof(Real) == 4 ? min(own, avail) * 3 / 4 : 0;
    const int per = max(1, NW / (nr - 1));
    for (int t = nown > 0 ? warp : 1 << 20; t < (nr - 1) * per; t += NW) {
      const int r = (rank + 1 + t % (nr - 1)) % nr, sub = t / (nr - 1);
      unsigned char *peer = cl.map_shared_rank(sm, r);
      for (int q = sub * 32 + lid; q < nA; q += per * 32) {
        const unsigned off = pl.A4 + (unsigned)sizeof(V) * lo + 16 * q;
        *(uint4 *)(peer + off) = *(const uint4 *)(sm + off);
      }
      for (int q = sub * 32 + lid; q < nL; q += per * 32) {
        const unsigned off = pl.L3 + 12 * lo + 16 * q;
        *(uint4 *)(peer + off) = *(const uint4 *)(sm + off);
      }
    }
    if (warp == 0) {
      const int2 m = make_int2(misc[MISC_DMAX], misc[MISC_NEAR_DISP]);
      __syncwarp();
      if (lid == 0) { misc[MISC_DMAX] = 0; misc[MISC_NEAR_DISP] = 0; }
      if (lid < nr) cl.map_shared_rank(dmax, lid)[par * SPLIT_MAX + rank] = m;
    }
  };

  unsigned ew_done = 0;   // count of the workers' forces of this step
  // ---- one evaluation of the forces, up to and including the second barrier
  const double cdist = a.lab_cdist[label], coefT = a.lab_coef[label];
  const Real rcd = (Real)(1.0 / cdist);
  // DH: the cutoff is scaled by the Debye length (force_ele_DH.F90:44); Ewald and Coulomb: in A
  const double cut = a.i_ele >= 2 ? a.cutoff_ele : a.cutoff_ele * cdist;
  const Real cut2 = (Real)(cut * cut);
  const Real ew_a = (Real)a.ewld_alpha, ew_a2 = (Real)(a.ewld_alpha * a.ewld_alpha), ew_b = (Real)a.ewld_beta;
  const int n_ts = (nts + 31) >> 5, n_hb = (nh + 7) >> 3, n_st = (nst + 15) >> 4, n_dh = (nrow + RW - 1) / RW;
  const int n_ex = (nown + 32 / SG - 1) / (32 / SG), n_ba = (nba + 31) >> 5, n_bd = (nbd + 31) >> 5, n_nz = (nown + 31) >> 5;
  const int c_ts = n_hb, c_st = c_ts + n_ts, c_dh = c_st + n_st, c_ex = c_dh + n_dh, c_ba = c_ex + n_ex,
            c_bd = c_ba + n_ba, c_nz = c_bd + n_bd;
  const Real ra = (Real)a.exv_adjust, ra2 = ra * ra, inv_ra2 = (Real)(1.0 / (a.exv_adjust * a.exv_adjust));
  const Real dist_ps = (Real)a.exv_dist_PS, dist_rr = (Real)a.exv_dist;
  int nclamp = 0;

  // force_exv_dt15.F90:204-265 for the pair (i, j): one 16-byte load screens
  // it; inside the screen radius the hi + lo difference is taken
  auto exv_pair = [&](int i, int j, int img, const V &pi, Real scr2, double &fx, double &fy, double &fz) SPLIT_INL {
    const V pj = s.A4[j];
    Real sx, sy, sz;
    pair_diff(pi, pj, img, sx, sy, sz);
    if (sq3(sx, sy, sz) > scr2) return;
    Real wx = sx, wy = sy, wz = sz;
    if constexpr (sizeof(Real) == 4) {
      wx = sx + (s.L3[3 * j] - s.L3[3 * i]); wy = sy + (s.L3[3 * j + 1] - s.L3[3 * i + 1]);
      wz = sz + (s.L3[3 * j + 2] - s.L3[3 * i + 2]);
    }
    const Real r2 = sq3(wx, wy, wz);
    const int ti = typ(i), ci = cls(i), tj = typ(j), cj = cls(j);
    const Real bix = s.RE[2 * i], bjx = s.RE[2 * j];
    // contact rule: 0 base-base / RNA-RNA, 1 phosphate-sugar, 2 radius sum (DT19: force_exv_dt15.F90:60-66)
    const int rule = a.dt19 ? ((ti == 3 && tj == 3) ? 0 : 2)
                            : (((ti == 2 && tj == 4) || (ti == 4 && tj == 2)) ? 1 : ((ci == 2 && cj == 2) ? 0 : 2));
    const Real dij = rule == 0 ? dist_rr : (rule == 1 ? dist_ps : bix + bjx);
    if (r2 > dij * dij) return;
    Real rinv = invsqrt(r2);
    Real dr = fma(r2, rinv, ra) - dij;
    if (sizeof(Real) == 4 && dr < (Real)1.5) {
      // the steep part of the potential: distance and dr in FP64 (see lane_kernel.cu)
      const double ex = (double)sx + ((double)s.L3[3 * j] - (double)s.L3[3 * i]);
      const double ey = (double)sy + ((double)s.L3[3 * j + 1] - (double)s.L3[3 * i + 1]);
      const double ez = (double)sz + ((double)s.L3[3 * j + 2] - (double)s.L3[3 * i + 2]);
      const double d64 = sqrt(sq3(ex, ey, ez));
      const double dij64 = rule == 0 ? a.exv_dist : (rule == 1 ? a.exv_dist_PS : (double)bix + (double)bjx);
      rinv = (Real)(1.0 / d64);
      dr = (Real)(d64 + a.exv_adjust - dij64);
    }
    const Real coef = s.RE[2 * i + 1] * s.RE[2 * j + 1];
    const Real ro2 = fdiv(ra2, dr * dr);
    const Real ro4 = ro2 * ro2, ro8 = mulr(ro4, ro4), ro14 = mulr(ro2 * ro4, ro8);
    Real f = fabs((Real)12 * coef * (ro14 - ro8) * dr * inv_ra2 * rinv);
    // DE_MAX clamp; each pair is visited from both beads and counted once
    if (f > (Real)50) { f = 50; nclamp += j > i; }
    fx -= (double)(f * wx); fy -= (double)(f * wy); fz -= (double)(f * wz);
  };

  // Electrostatic force of row bead i on its partner entry e (bead and
  // image); KIND 0 Debye-Hueckel, 1 Coulomb, 2 Ewald real space, 3
  // Debye-Hueckel with Mg-P pairs on the PMF table
  auto ele_pair = [&](auto kind, int i, int e, const V &pi, Real qci, const double *pmf_row, Real &ax, Real &ay,
                      Real &az) SPLIT_INL {
    constexpr int KIND = decltype(kind)::value;
    const int j = PER ? (e & ((1 << SP_IMG) - 1)) : e;
    const V pj = s.A4[j];
    Real x, y, z;
    pair_diff(pi, pj, PER ? e >> SP_IMG : 0, x, y, z);
    const Real r2 = sq3(x, y, z);
    const Real ri = invsqrt(r2);
    const Real d = r2 * ri;
    Real f;
    if constexpr (KIND == 1) {
      f = qci * pj.w * ri * ri * ri;   // force_ele_coulomb.F90:66-71 (no clamp)
    } else if constexpr (KIND == 2) {
      // force_ele_coulomb_ewld.F90:118-137 (no clamp); pairs past the cutoff add nothing
      f = (r2 <= cut2) ? qci * pj.w * fma((Real)erfc(ew_a * d), ri, mulr(ew_b, (Real)exp(-ew_a2 * r2))) * ri * ri : (Real)0;
    } else {
      f = qci * pj.w * ri * ri * (ri + rcd) * fexp<Real>(-d * rcd);   // force_ele_DH.F90:72-117
      if (KIND == 3 && pmf_row && j != np && mg_p_pair(typ(i), typ(j)) && (double)d <= a.pmf_rmax) {
        bool low = false;
        f = (Real)pmf_row[pmf_bin(a, (double)d, low)] * ri;
        if (low) misc[MISC_PMF] = 1;
      }
    }
    if (!(r2 <= cut2)) f = 0;
    if ((KIND == 0 || KIND == 3) && f > (Real)50) { f = 50; nclamp += j > i; }   // DE_MAX, counted from the lower bead
    ax -= f * x; ay -= f * y; az -= f * z;
  };
  // the forces of RW charged rows, LQ threads each, to the beads' owners
  auto ele_rows = [&](auto kind, int k) SPLIT_INL {
    constexpr int KIND = decltype(kind)::value;
    const int gq = lid & (LQ - 1);
    double fx = 0, fy = 0, fz = 0;
    int i = 0;
    if (k < nrow) {
      i = qb[kq_lo + k];
      const V pi = s.A4[i];
      const Real qci = (Real)((double)pi.w * coefT);
      const double *pmf_row = nullptr;
      if (KIND == 3 && (typ(i) == 2 || typ(i) == 5)) pmf_row = a.pmf_f + (size_t)label * a.pmf_nbin;
      Real ax = 0, ay = 0, az = 0, bx = 0, by = 0, bz = 0;   // two pairs in flight
      if (misc[MISC_ELIST]) {
        const uint32_t *lst = (const uint32_t *)elist;   // two entries per word
        const int n = eoff[k + 1] >> 1;
        for (int e = (eoff[k] >> 1) + gq; e < n; e += LQ) {
          const uint32_t p = lst[e];
          ele_pair(kind, i, (int)(p & 0xffffu), pi, qci, pmf_row, ax, ay, az);
          ele_pair(kind, i, (int)(p >> 16), pi, qci, pmf_row, bx, by, bz);
        }
      } else {
        // lists too long for the shared memory: the bits of the row, the same
        // entries in the same order as above (2 (gq + LQ r) and the one after)
        int w = 0, n = 0;   // word, bits of the words before
        uint32_t m = mele[k * W];
        auto entry = [&](int e) SPLIT_INL {   // bead (and image) of entry e >= n, -1 beyond the last
          int c;
          while (n + (c = __popc(m)) <= e) {
            if (++w >= W) return -1;
            n += c;
            m = mele[k * W + w];
          }
          const int j = (w << 5) + nth_bit(m, e - n);
          return PER ? (j | split_image(a, s, i, j) << SP_IMG) : j;
        };
#pragma unroll 1
        for (int e = 2 * gq;; e += 2 * LQ) {
          const int p = entry(e);
          if (p < 0) break;
          ele_pair(kind, i, p, pi, qci, pmf_row, ax, ay, az);
          const int q = entry(e + 1);
          if (q < 0) break;
          ele_pair(kind, i, q, pi, qci, pmf_row, bx, by, bz);
        }
      }
      fx = (double)ax + (double)bx; fy = (double)ay + (double)by; fz = (double)az + (double)bz;
    }
    for (int o = LQ >> 1; o > 0; o >>= 1) {
      fx += __shfl_xor_sync(0xffffffffu, fx, o); fy += __shfl_xor_sync(0xffffffffu, fy, o);
      fz += __shfl_xor_sync(0xffffffffu, fz, o);
    }
    if (k < nrow && gq < 3) {
      const int r = (int)__umulhi((unsigned)i, magic);
      const double f = gq == 0 ? fx : (gq == 1 ? fy : fz);
      double *o = dhF + 3 * (i - r * own) + gq;
      if (r == rank) *o = f;
      else *cl.map_shared_rank(o, r) = f;
    }
  };

  auto sweep = [&](long long istep, int noise_step, int par, bool rec) SPLIT_INL {
    const int f_exc = MISC_EXCESS + par;
    // flags of the next step: their last readers passed the barrier before this sweep, and
    // they are set only behind the one after it
    if (tid == 0) misc[MISC_EXCESS + (par ^ 1)] = 0;
    const int c_end = c_nz + (noise_step >= 0 ? n_nz : 0);
    int c = warp;
    while (c < c_end) {
      int cn = 0;   // the next chunk, requested before this one is processed
      if (lid == 0) cn = atomicAdd(&misc[MISC_CHUNK], 1);
      if (c >= c_ex && c < c_ba) {
        // exv of 32 / SG own beads, SG threads each: thread g takes the
        // partners j with j % SG == g, in ascending order.  A recording pass
        // keeps those within the screen radius + SP_SKIN; later passes
        // visit only these (partners further off add nothing, so the sums
        // are the same bits)
        const int li = (c - c_ex) * (32 / SG) + lid / SG, i = lo + li;
        const bool valid = li < nown;
        double fx = 0, fy = 0, fz = 0;
        if (valid) {
          const V pi = s.A4[i];
          const Real sr = scr[li], scr2 = sr * sr;
          uint16_t *lst = near + (li * SG + g) * SP_NEAR;
          int n = ncnt[li * SG + g], w = 0;
          const bool scan = rec || n == 0xFF;
          bool more = scan, first = true;
          uint32_t m = 0;
          do {
            if (scan) {   // the next (at most SP_NEAR) near partners from the row's bits
              const Real nscr = sr + (Real)SP_SKIN, nscr2 = nscr * nscr;
              for (n = 0; n < SP_NEAR;) {
                while (m == 0 && w < W) m = mexv[li * W + w++] & (0x01010101u << g);
                if (m == 0) { more = false; break; }
                const int j = ((w - 1) << 5) + __ffs(m) - 1;
                m &= m - 1;
                const V pj = s.A4[j];
                Real x = pj.x - pi.x, y = pj.y - pi.y, z = pj.z - pi.z;
                int img = 0;
                if (PER) {   // far in the nearest image is far in the pair's own
                  Real cx = fabs(x), cy = fabs(y), cz = fabs(z);
                  cx = min(cx, (Real)fabs((Real)a.psize[0] - cx)); cy = min(cy, (Real)fabs((Real)a.psize[1] - cy));
                  cz = min(cz, (Real)fabs((Real)a.psize[2] - cz));
                  if (sq3(cx, cy, cz) > nscr2 + (Real)0.1) continue;
                  img = split_image(a, s, i, j);
                  pair_diff(pi, pj, img, x, y, z);
                }
                if (sq3(x, y, z) <= nscr2) lst[n++] = (uint16_t)(PER ? (j | (img << SP_IMG)) : j);
              }
              if (rec && first) {
                ncnt[li * SG + g] = (uint8_t)(more ? 0xFF : n);
                if (g == 0) NR4[li] = make_float4((float)pi.x, (float)pi.y, (float)pi.z, 0.f);
              }
              first = false;
            }
            for (int k = 0; k < n; ++k) {
              const int e = lst[k];
              exv_pair(i, PER ? (e & ((1 << SP_IMG) - 1)) : e, PER ? e >> SP_IMG : 0, pi, scr2, fx, fy, fz);
            }
          } while (more);
        }
        group_reduce<Real>(fx, fy, fz, SG);
        if (valid && g < 3) exF[3 * li + g] = g == 0 ? fx : (g == 1 ? fy : fz);
      } else if (c >= c_dh && c < c_ex) {
        const int k = (c - c_dh) * RW + lid / LQ;
        if (PER && ewald) ele_rows(std::integral_constant<int, PER ? 2 : 0>(), k);
        else if (coul) ele_rows(std::integral_constant<int, 1>(), k);
        else if (PER && a.pmf_f) ele_rows(std::integral_constant<int, PER ? 3 : 0>(), k);
        else ele_rows(std::integral_constant<int, 0>(), k);
      } else if (c >= c_st && c < c_dh) {
        // 16 stacks, two threads each (one dihedral per thread)
        const int k0 = ((c - c_st) << 4) + (lid >> 1), role = lid & 1, k = min(k0, nst - 1);
        const uint4 ix = *(const uint4 *)(sm + pl.sti + 16 * k);
        const uint32_t *dw = (const uint32_t *)(sm + pl.std_) + 7 * k;
        const Real *cf = (const Real *)(sm + pl.stc) + 6 * k;   // nat (3), coef (3)
        const int m[7] = {(int)(ix.x & 0xffff), (int)(ix.x >> 16), (int)(ix.y & 0xffff), (int)(ix.y >> 16),
                          (int)(ix.z & 0xffff), (int)(ix.z >> 16), (int)(ix.w & 0xffff)};
        const double u0 = u0s[k];
        const bool off = T.ntst > 0 && stack_excluded<Real>(a, T, split_view(s, magic), stk[k]), live = k0 < nst;
        // the stack in W (nat and coef of its distance, then of this thread's
        // dihedral): forces of beads 0 / 1, 2 / 6, 3 / 5 and (thread 0) 4;
        // true when a triple is too straight for FP32
        auto stack = [&](bool mine, auto w, auto n0, auto k1, auto nat, auto kd) SPLIT_INL {
          typedef decltype(w) Wt;
          const R3<Wt> v21 = rvec(Wt(), m[0], m[1]), v54 = rvec(Wt(), m[3], m[4]), v56 = rvec(Wt(), m[5], m[4]);
          const R3<Wt> u = rvec(Wt(), role ? m[5] : m[3], role ? m[6] : m[2]);
          const Dih<Wt> o = dihedral<Wt, false>(u, sel3(role != 0, v56, v54), sel3(role != 0, v54, v56), nat, kd, (Wt)1);
          const int other = __shfl_xor_sync(0xffffffffu, (int)o.straight, 1);   // every lane takes part
          Wt dist, rdist;
          length(sdot(v21, v21), dist, rdist);
          const Wt dd = dist - n0;
          const Wt ediv = (Wt)1 + k1 * dd * dd + (o.e + __shfl_xor_sync(0xffffffffu, o.e, 1));
          const R3<Wt> fb = add3(o.b, shx3(o.d, 1)), fc = add3(o.c, shx3(o.c, 1));
          const Wt gd = (Wt)2 * k1 * (dd * rdist);
          const Wt pre = off ? (Wt)0 : (Wt)(u0 / ((double)ediv * (double)ediv));
          const bool bad = o.straight || other != 0;
          if (mine && (!bad || off)) {
            auto put = [&](int q, R3<Wt> f) SPLIT_INL {
              put_word(slots, rank, dw[q], R3<Real>{(Real)f.x, (Real)f.y, (Real)f.z});
            };
            put(role, mul3(role ? pre * gd : -(pre * gd), v21));
            put(role ? 6 : 2, mul3(pre, o.a));
            put(role ? 5 : 3, mul3(pre, fb));
            if (role == 0) put(4, mul3(pre, fc));
          }
          return bad && !off && mine;
        };
        const bool bad = stack(live, (Real)0, cf[0], cf[3], cf[1 + role], cf[4 + role]);
        if constexpr (sizeof(Real) == 4)
          if (__any_sync(0xffffffffu, bad)) {   // those in FP64, from the FP64 tables (see term_stack)
            const double *nd = a.st_nat + 3 * (size_t)(T.st0 + stk[k]), *cd = a.st_coef + 3 * (size_t)(T.st0 + stk[k]);
            stack(bad, 0.0, ldro(nd), ldro(cd), ldro(nd + 1 + role), ldro(cd + 1 + role));
          }
      } else if (c >= c_ba && c < c_bd) {
        const int k = ((c - c_ba) << 5) + lid;   // force_bangle.F90:103-147
        if (k < nba) {
          const uint2 ix = *(const uint2 *)(sm + pl.bai + 8 * k);
          const uint32_t *dw = (const uint32_t *)(sm + pl.bad) + 3 * k;
          const Real nat = ((const Real *)(sm + pl.bac))[2 * k], cf = ((const Real *)(sm + pl.bac))[2 * k + 1];
          const int m1 = (int)(ix.x >> 16);
          const R3<Real> v21 = rvec(Real(), (int)(ix.x & 0xffff), m1), v32 = rvec(Real(), m1, (int)ix.y);
          R3<Real> f[3];
          split_angle<Real>(v21, v32, nat, cf, f);
#pragma unroll
          for (int p = 0; p < 3; ++p) put_word(slots, rank, dw[p], f[p]);
        }
      } else if (c >= c_bd && c < c_nz) {
        const int k = ((c - c_bd) << 5) + lid;   // force_bond.F90:41-56
        if (k < nbd) {
          const uint32_t ix = ((const uint32_t *)(sm + pl.bdi))[k];
          const uint32_t *dw = (const uint32_t *)(sm + pl.bdd) + 2 * k;
          const Real nat = ((const Real *)(sm + pl.bdc))[2 * k], cf = ((const Real *)(sm + pl.bdc))[2 * k + 1];
          const R3<Real> v = rvec(Real(), (int)(ix & 0xffff), (int)(ix >> 16));
          Real dist, rdist;
          length(sdot(v, v), dist, rdist);
          const Real f = cf * ((Real)-2.0 * ((dist - nat) * rdist));
          put_word(slots, rank, dw[0], mul3(-f, v));
          put_word(slots, rank, dw[1], mul3(f, v));
        }
      } else if (c >= c_nz) {
        const int li = ((c - c_nz) << 5) + lid;
        if (li < nown) noise3(a, lane, L, lo + li, istep, noise_step, NZ[li], NZ[OS + li], NZ[2 * OS + li]);
      } else if (c < n_hb) {
        // 8 hydrogen bonds (force_dtrna_hbond15.F90:91-353), four threads
        // each: one dihedral on each of threads 0..2, the angles on 0 and 1,
        // the distance on 2
        const int k0 = (c << 3) + (lid >> 2), role = lid & 3, k = min(k0, nh - 1), h = hbk[k];
        const uint32_t *ix = (const uint32_t *)(sm + pl.hbi) + 3 * k, *dw = (const uint32_t *)(sm + pl.hbd) + 6 * k;
        const Real *cf = (const Real *)(sm + pl.hbc) + 13 * k;   // nat (6), coef (7)
        const int m[6] = {(int)(ix[0] & 0xffff), (int)(ix[0] >> 16), (int)(ix[1] & 0xffff), (int)(ix[1] >> 16),
                          (int)(ix[2] & 0xffff), (int)(ix[2] >> 16)};
        const uint8_t f = k0 < nh ? hbf[k] : (uint8_t)0;
        const R3<Real> v12 = bvec(std::true_type(), Real(), m[1], m[0]);
        Real a12, r12;
        length(sdot(v12, v12), a12, r12);
        const Real d12 = a12 - cf[0];
        const bool act = (f & 1) && !(fabs((double)d12) > a.hb_cutoff_dist);
        Real e = 0;
        if (__any_sync(0xffffffffu, act)) {
          auto dv = [&](int p, int q) SPLIT_INL { return bvec(std::true_type(), Real(), q, p); };   // x_p - x_q
          const Real MAXC = (Real)a.max_abscos;
          const R3<Real> v13 = dv(m[0], m[2]), v42 = dv(m[3], m[1]);
          const R3<Real> ve = dv(role == 1 ? m[4] : m[3], role == 1 ? m[2] : m[5]);   // v53 or v46
          // dihedrals 4-2=1=3, 5-3-1=2 and 1=2-4-6
          const bool r1 = role == 1, r2 = role >= 2;
          const R3<Real> u = sel3(r1, ve, sel3(r2, v12, v42)), w = sel3(r1, v13, sel3(r2, v42, v12)),
                         z = sel3(r1, v12, sel3(r2, ve, v13));
          Dih<Real> o = dihedral<Real, true>(u, w, z, cf[3 + min(role, 2)], cf[10 + min(role, 2)], MAXC);
          // angles 3-1=2 (vectors v13, v12) and 1=2-4 (v12, v42, opposite sign)
          const R3<Real> p = sel3(r1, v12, v13), q = sel3(r1, v42, v12);
          const Real p2 = sdot(p, p), q2 = sdot(q, q), pq = sdot(p, q);
          Real apq, co, cp, cq;   // |p| |q|, the cosine, pq / p2, pq / q2
          if constexpr (sizeof(Real) == 8) {
            Real r;
            length(p2 * q2, apq, r);
            const Real r2 = r * r;
            co = quot(pq, apq, r); cp = quot(pq, p2, q2 * r2); cq = quot(pq, q2, p2 * r2);
          } else {
            apq = sqrt(p2) * sqrt(q2); co = fdiv(pq, apq); cp = fdiv(pq, p2); cq = fdiv(pq, q2);
          }
          const Real pqc = fabs(co) > MAXC ? (Real)copysign(apq * MAXC, co) : pq;
          const Real da = acos(co > (Real)1 ? (Real)1 : (co < (Real)-1 ? (Real)-1 : co)) - cf[r1 ? 2 : 1], ca = role < 2 ? cf[r1 ? 9 : 8] : (Real)0;
          const Real pre = (r1 ? (Real)-2 : (Real)2) * ca * da * invsqrt(det2(p2, q2, pqc, pqc));
          const bool live = role < 2;   // threads 2 and 3 add no angle term (their angle may be capped to 0 / 0)
          const R3<Real> zero{0, 0, 0};
          const R3<Real> A{fma(-cp, p.x, q.x), fma(-cp, p.y, q.y), fma(-cp, p.z, q.z)};
          const R3<Real> B{fma(-cq, q.x, p.x), fma(-cq, q.y, p.y), fma(-cq, q.z, p.z)};
          const R3<Real> fi = live ? mul3(pre, A) : zero, fk = live ? mul3(pre, B) : zero;
          const R3<Real> fik = live ? mul3(-pre, add3(A, B)) : zero;
          Real ex = -o.e;
          if (role < 2) ex -= mulr(mulr(ca, da), da);
          if (role == 2) ex -= mulr(mulr(cf[7], d12), d12);
          if (role == 3) { ex = 0; o.a = o.b = o.c = o.d = zero; }
          const Real gd = role == 2 ? (Real)2 * cf[7] * d12 * r12 : (Real)0;
          // the thread's share of the forces of beads 1..4 (5 is thread 1's alone, 6 thread 2's)
          R3<Real> b1 = add3(add3(r2 ? o.a : o.c, r1 ? fi : fik), mul3(gd, v12));
          R3<Real> b2 = add3(add3(r1 ? o.d : o.b, r1 ? fik : fk), mul3(-gd, v12));
          R3<Real> b3 = add3(role == 0 ? o.d : (r1 ? o.b : zero), r1 ? zero : fi);
          R3<Real> b4 = add3(role == 0 ? o.a : (r1 ? zero : o.c), r1 ? fk : zero);
          // sums over the four threads, scattered: thread r ends with bead r + 1
          const bool up = (role & 2) != 0, odd = (role & 1) != 0;
          R3<Real> s0 = sel3(up, b3, b1), s1 = sel3(up, b4, b2);
          s0 = add3(s0, shx3(sel3(up, b1, b3), 2));
          s1 = add3(s1, shx3(sel3(up, b2, b4), 2));
          R3<Real> tot = sel3(odd, s1, s0);
          tot = add3(tot, shx3(sel3(odd, s0, s1), 1));
          ex += __shfl_xor_sync(0xffffffffu, ex, 1);
          ex += __shfl_xor_sync(0xffffffffu, ex, 2);
          e = cf[6] * exp(ex);
          if (act) {
            put_word(slots, rank, dw[role], mul3(e, tot));
            if (role == 1) put_word(slots, rank, dw[4], mul3(e, o.a));
            if (role == 2) put_word(slots, rank, dw[5], mul3(e, o.d));
            if (role < 3) {   // hbond-site counters, on the first CTA
              int *exc0 = cl.map_shared_rank(exc, 0);
#pragma unroll
              for (int t = 0; t < 2; ++t) {
                const uint32_t sv = ((const uint32_t *)(sm + pl.hbs))[6 * k + 2 * role + t];   // site | valence << 24
                if (sv != 0xffffffffu && atomicAdd(&exc0[sv & 0xffffffu], 1) + 1 > (int)(sv >> 24))
                  for (int r = 0; r < nr; ++r) cl.map_shared_rank(misc, r)[f_exc] = 1;
              }
            }
          }
        }
        if (k0 < nh) {
          if (!act && (f & 2)) {   // the slots of the last force
            const R3<Real> zero{0, 0, 0};
            put_word(slots, rank, dw[role], zero);
            if (role < 2) put_word(slots, rank, dw[4 + role], zero);
          }
          if (role == 0) {
            hbf[k] = (uint8_t)((f & 1) | (act ? 2 : 0));
            a.hb_flag[L.hb0 + h] = (uint8_t)((f & 1) | (act ? 2 : 0));
            a.hb_ene[L.hb0 + h] = act ? (double)e : 0.0;
          }
        }
      } else {
        const int k = ((c - c_ts) << 5) + lid;
        if (k < nts) {
          const SplitView<Real> s2 = split_view(s, magic);   // copies: the values used elsewhere stay in registers
          const TopDesc T2 = T;
          const SplitDst<Real> d2 = dst;
          term_tstack<Real>(a, T2, s2, d2, tsk[k]);
        }
      }
      c = __shfl_sync(0xffffffffu, cn, 0);
    }
    if constexpr (PER)
      if (a.ew_nwork && warp == 0) ew_wait(a, EWS_DONE, ew_done);   // this step's reciprocal forces
    cl.sync();
    if (tid == 0) {
      misc[MISC_CHUNK] = NW;   // every warp has taken its last chunk
      misc[MISC_NEAR_BAD] = 0;
    }
    if (misc[f_exc]) {   // the same in every CTA
      if (tid == 0 && rank == 0) {
        const double beta = a.hb_beta_global ? (a.rex ? a.rex->beta_global : a.beta_hbond15) : a.lab_beta[label];
        prune_hbonds<Real>(a, lane, L, T, istep, beta, true, exc, [&](int h) {
          const int *m = a.hb_idx + 6 * (size_t)(T.hb0 + h);
          for (int q = 0; q < 6; ++q) put_slot<Real>(dst, T.slot_hb + 6 * (size_t)h + q, ldro(m + q), 0, 0, 0);
        });
      }
      cl.sync();
    }
  };

  // ---- the steps (each phase has one place in the code, so that it is
  // inlined): [rebuild] - [x update of every own bead] - barrier - sweep -
  // barrier - force sums, v / a update and, unless the lists are rebuilt
  // first, the next x update
  auto cadence = [&](long long is) SPLIT_INL { return (is % a.n_step_neighbor) == 1 || is == 1; };
  if (!lists_new) { expand_rows(); __syncthreads(); }
  const bool stepping = a.mode == KM_STEP || a.mode == KM_XSTEP || a.mode == KM_VSTEP || a.mode == KM_VXSTEP;
  const bool first_x = a.mode == KM_STEP || a.mode == KM_XSTEP;
  const int nloop = a.mode == KM_STEP ? lane_steps : (a.mode == KM_XSTEP || a.mode == KM_NEIGHBOR ? 0 : 1);
  // trigger of the launch's first x update, from the dxyz loaded
  bool fire = false;
  if (first_x || a.mode == KM_VXSTEP) {
    if (skin) fire = skin_exact(true);
    else fire = cadence(istep0 + 1 + (first_x ? 0 : 1));
  }
  long long istep = istep0;          // the step whose forces come next (stepping: counted from the first x update)
  if (stepping) istep = istep0 + 1;
  bool do_build = lists_new || (first_x && fire), do_x = first_x;
  for (int step = 0;; ++step) {
    const int par = (int)(istep & 1);
    if (do_build) build(istep, step == 0);
    if (do_x) {
      for (int l0 = 0; l0 < nown; l0 += NG) xmove(l0 + grp, l0 + grp < nown, fire);
      send(par);
    }
    if (step >= nloop) break;
    // dxyz_mp = 0 (time_integral_pre.F90:79)
    if (a.mode == KM_PRE && skin) for (int q = tid; q < 3 * OS; q += NT) Dv[q] = 0.0;
    if constexpr (PER)
      if (a.ew_nwork) {   // (behind send's barrier)
        ew_done = (unsigned)(step + 1) * (unsigned)a.ew_nwork;
        ew_publish(a, s.PX, np, lo, nown, L.state0, tid, NT);
      }
    cl.sync();   // the positions of this step are complete
    if constexpr (PER)
      if (a.ew_nwork && tid == 0) ew_signal(a, EWS_READY);
    const bool next = a.mode == KM_STEP ? step + 1 < nloop
                                        : (a.mode == KM_VXSTEP && (!a.lane_nsteps || a.step_k + 1 < a.lane_nsteps[lane]));
    // trigger of the next step's x update
    if (next && a.mode == KM_STEP) {
      if (!skin) fire = cadence(istep + 1);
      else {
        const int M = __reduce_max_sync(0xffffffffu, lid < nr ? dmax[par * SPLIT_MAX + lid].x : 0);
        fire = 2.0f * sqrtf(__int_as_float(M)) >= (float)a.neigh_margin * 0.9999f && skin_exact(false);
      }
    }
    // the near lists are recorded anew, by every CTA: after a build or a
    // launch, or when a bead has moved too far since
    const int far = __reduce_max_sync(0xffffffffu, lid < nr ? dmax[par * SPLIT_MAX + lid].y : 0);
    const bool rec = misc[MISC_NEAR_BAD] != 0 || __int_as_float(far) > SP_SKIN_DISP * SP_SKIN_DISP;
    sweep(istep, stepping ? a.noise_base + step : (a.mode == KM_PRE ? a.noise_base : -1), par, rec);
    const bool move = next && !fire;
    for (int l0 = 0; l0 < nown; l0 += NG) {
      const int li = l0 + grp, i = lo + li;
      const bool valid = li < nown;
      double fx = 0, fy = 0, fz = 0;
      // the reciprocal-space force (from L2: other SMs wrote it)
      const double fe = (PER && a.f_ext && valid && g < 3) ? __ldcg(a.f_ext + 3 * (size_t)(L.state0 + i) + g) : 0.0;
      if (valid)
        for (int p = iptr[li] + g; p < iptr[li + 1]; p += SG) {
          fx += (double)slots[3 * p]; fy += (double)slots[3 * p + 1]; fz += (double)slots[3 * p + 2];
        }
      group_reduce<Real>(fx, fy, fz, SG);
      if (valid && g < 3) {
        double f = (g == 0 ? fx : (g == 1 ? fy : fz)) + exF[3 * li + g] + dhF[3 * li + g];
        if (PER) f += fe;
        const int q = g * OS + li;
        if (a.mode == KM_FORCE) {
          a.out_force[3 * (size_t)(L.state0 + i) + g] = f;
        } else {
          // time_integral.F90:169-183 (KM_PRE: a(0)), each product rounded as the reference evaluates it
          const double acc = smad<Real>(f, RC[li], C1[li], NZ[q]);
          if (stepping) Vv[q] = smad<Real>(C2[li], Vv[q], C3[li], __dadd_rn(Av[q], acc));
          Av[q] = acc;
          if (stepping && !(f == f)) misc[MISC_NAN] = 1;
        }
      }
      __syncwarp();
      if (move) xmove(li, valid, false);
    }
    if (move) send(par ^ 1);
    // hbond-site counters of the next sweep (read behind this one's barriers)
    if (rank == 0) for (int k = tid; k < T.nsite; k += NT) exc[k] = 0;
    if (!next) break;
    ++istep;
    do_build = do_x = fire;
    if (fire) __syncthreads();
    if (a.mode == KM_VXSTEP && !fire) break;
  }
  // KM_VXSTEP counts the step whose forces it took, not the x update that follows
  const long long istep_end = !stepping || a.mode == KM_XSTEP ? istep0 : (a.mode == KM_STEP ? istep : istep0 + 1);
  cl.sync();   // no distributed shared-memory access after this
  // ---- write back the own beads
  if (a.mode != KM_FORCE) {
    for (int q = tid; q < 3 * nown; q += NT) {
      const int li = q / 3, d = q - 3 * li, i = lo + li;
      const size_t o = 3 * (size_t)(L.state0 + lo) + q;
      a.xyz[o] = s.X[d * np + i];
      a.pxyz[o] = s.PX[d * np + i];
      if (PER) a.p0xyz[o] = s.QX[d * np + i];
      a.velo[o] = Vv[d * OS + li]; a.accel[o] = Av[d * OS + li];
      if (skin) a.dxyz[o] = Dv[d * OS + li];
    }
  }
  if (nclamp) atomicAdd(&misc[MISC_CLAMP], nclamp);
  __syncthreads();
  if (tid == 0) {
    if (misc[MISC_CLAMP]) atomicAdd((unsigned long long *)&st.nclamp, (unsigned long long)misc[MISC_CLAMP]);
    if (misc[MISC_NAN]) atomicOr(&st.flags, LF_NAN);
    if (misc[MISC_PMF]) atomicOr(&st.flags, LF_PMF);
    if (!misc[MISC_ELIST]) atomicOr(&st.flags, LF_ROW_BITS);
    if (PER && a.ew_nwork && rank == 0 && __ldcg(a.ew_sync + EWS_ABORT)) atomicOr(&st.flags, LF_WAIT);
    if (rank == 0) st.istep = istep_end;
  }
}


} // namespace tis
