// lane_common.cuh -- device helpers shared by the kernels that step lanes
// (lane_kernel.cu: a lane on one CTA or a pair; split_kernel.cuh: a lane
// split over a larger cluster).
#pragma once
#include "device_common.cuh"

namespace tis {

// ------------------------------------------------------------ skin rule
// time_integral.F90:57-93: rebuild when sqrt(d2max) + sqrt(d2max_2nd) >
// neigh_margin, d2 = dot_product(dxyz_mp, dxyz_mp) of each bead.  The pair
// (d2max, d2max_2nd) is the top two of the multiset of d2 values, so partial
// results merge exactly in any order: each warp folds its beads, every warp
// then folds the per-warp pairs (of both CTAs of a cluster) and reaches the
// same decision without another barrier.
__device__ __forceinline__ void top2_add(double &m1, double &m2, double d2) {
  if (d2 > m1) { m2 = m1; m1 = d2; } else if (d2 > m2) m2 = d2;
}
__device__ __forceinline__ void top2_merge(double &m1, double &m2, double o1, double o2) {
  const double n1 = fmax(m1, o1), n2 = fmax(fmin(m1, o1), fmax(m2, o2));
  m1 = n1; m2 = n2;
}
__device__ __forceinline__ void top2_warp(double &m1, double &m2) {
  for (int o = 16; o > 0; o >>= 1) {
    const double o1 = __shfl_xor_sync(0xffffffffu, m1, o), o2 = __shfl_xor_sync(0xffffffffu, m2, o);
    top2_merge(m1, m2, o1, o2);
  }
}
// dot_product(dxyz, dxyz) in the Fortran operation order, no contraction
__device__ __forceinline__ double disp2(double x, double y, double z) {
  return __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z));
}
// per-warp pair of this thread's (m1, m2) into red[2 w], red[2 w + 1]; every
// thread of the CTA calls it
__device__ __forceinline__ void top2_store(double m1, double m2, double *red) {
  top2_warp(m1, m2);
  if ((threadIdx.x & 31) == 0) { red[2 * (threadIdx.x >> 5)] = m1; red[2 * (threadIdx.x >> 5) + 1] = m2; }
}
// sqrt(d2max) + sqrt(d2max_2nd) > margin from every lane's pair (the
// decision is the same in every lane)
__device__ __forceinline__ bool skin_decide(double m1, double m2, double margin) {
  top2_warp(m1, m2);
  // FP32 screen: the float sum is within ~4e-7 (relative) of the FP64 one,
  // so outside a 1e-4 band around the margin it decides the same way
  const float sf = sqrtf((float)m1) + sqrtf((float)m2), mf = (float)margin;
  if (sf < mf * 0.9999f) return false;
  if (sf > mf * 1.0001f) return true;
  return __dadd_rn(sqrt(m1), sqrt(m2)) > margin;
}
// The trigger from the d2 of every bead (DD) and M, their maximum rounded
// up to float: M rules the skin out while 2 sqrt(M) is 1e-4 below the
// margin (sqrt(d2max) + sqrt(d2max_2nd) <= 2 sqrt(M)); else every warp
// takes the top two d2 of DD.  Every thread reaches the same decision.
__device__ __forceinline__ bool skin_trigger(int Mbits, const double *DD, int N, double margin) {
  const float M = __int_as_float(Mbits);
  if (2.0f * sqrtf(M) < (float)margin * 0.9999f) return false;
  double m1 = 0.0, m2 = 0.0;
  for (int b = (threadIdx.x & 31); b < N; b += 32) top2_add(m1, m2, DD[b]);
  return skin_decide(m1, m2, margin);
}
// the trigger from the per-warp pairs of this CTA (lanes 0 .. nwarp - 1) and,
// with two CTAs, of the other one (lanes 16 .. 16 + nwarp - 1, nwarp <= 16)
__device__ __forceinline__ bool skin_fires(const double *red, const double *peer_red, int nwarp, double margin) {
  const int lid = threadIdx.x & 31;
  double m1 = 0.0, m2 = 0.0;
  if (lid < nwarp) { m1 = red[2 * lid]; m2 = red[2 * lid + 1]; }
  else if (peer_red && lid >= 16 && lid - 16 < nwarp) { m1 = peer_red[2 * (lid - 16)]; m2 = peer_red[2 * (lid - 16) + 1]; }
  return skin_decide(m1, m2, margin);
}

// a b + c d of the integration: in the FP64 path each product rounded as
// the reference evaluates it (no contraction), so the update is the
// reference's to the last bit; the mixed path lets the compiler contract
template <typename Real>
__device__ __forceinline__ double mad2(double a, double b, double c, double d) {
  if constexpr (sizeof(Real) == 8) return __dadd_rn(__dmul_rn(a, b), __dmul_rn(c, d));
  else return a * b + c * d;
}
template <typename Real>
__device__ __forceinline__ double add_rn(double a, double b) {
  if constexpr (sizeof(Real) == 8) return __dadd_rn(a, b);
  else return a + b;
}

__device__ __forceinline__ void rebuild_counts(LaneState &st, int nexv, int nele, long long istep) {
  st.nrebuild++;
  st.last_rebuild = istep;
  st.nexv = nexv;
  st.nele = nele;
}


// exp for the Debye-Hueckel factor: FP64 in the FP64 path; the fast
// single-precision exponential in the mixed path (relative error about
// |x| 2^-22 for the arguments here, |x| <= 25)
template <typename Real> __device__ __forceinline__ Real fexp(Real x);
template <> __device__ __forceinline__ double fexp<double>(double x) { return exp(x); }
template <> __device__ __forceinline__ float fexp<float>(float x) { return __expf(x); }

template <typename Real>
__device__ __forceinline__ void group_reduce(double &fx, double &fy, double &fz, int G) {
  for (int o = G >> 1; o > 0; o >>= 1) {
    fx += __shfl_xor_sync(0xffffffffu, fx, o, G);
    fy += __shfl_xor_sync(0xffffffffu, fy, o, G);
    fz += __shfl_xor_sync(0xffffffffu, fz, o, G);
  }
}

__device__ __forceinline__ int pow2_floor_clamp(int x, int hi) {
  int g = 1;
  while (g * 2 <= x && g * 2 <= hi) g *= 2;
  return g;
}

// Periodic image of the pair fixed at the last rebuild (d_mirror(:, imirror)
// of the canonical (min, max) orientation, negated for the reverse one),
// recomputed from the positions wrapped at that rebuild with the same
// rounded FP64 operations as the list build: the same image as its mirror
// table, without a global-memory lookup.
template <typename T, typename S>
__device__ __forceinline__ void mirror_shift(const KArgs &a, const S &s, int i, int j, T &w0, T &w1, T &w2) {
  const int lo = i < j ? i : j, hi = i < j ? j : i;
  const T sg = (j > i) ? (T)1 : (T)-1;
  const double v0 = __dsub_rn(s.QX[hi], s.QX[lo]), v1 = __dsub_rn(s.QY[hi], s.QY[lo]),
               v2 = __dsub_rn(s.QZ[hi], s.QZ[lo]);
  if (v0 > a.psizeh[0]) w0 -= sg * (T)a.psize[0]; else if (v0 < -a.psizeh[0]) w0 += sg * (T)a.psize[0];
  if (v1 > a.psizeh[1]) w1 -= sg * (T)a.psize[1]; else if (v1 < -a.psizeh[1]) w1 += sg * (T)a.psize[1];
  if (v2 > a.psizeh[2]) w2 -= sg * (T)a.psize[2]; else if (v2 < -a.psizeh[2]) w2 += sg * (T)a.psize[2];
}

template <typename Real> __device__ __forceinline__ Real rsq(Real x);
template <> __device__ __forceinline__ double rsq<double>(double x) { return 1.0 / sqrt(x); }
template <> __device__ __forceinline__ float rsq<float>(float x) { return rsqrtf(x); }

} // namespace tis
