// split_ewald.cuh -- reciprocal-space Ewald forces inside the launch of the
// split lanes (split_kernel.cuh): all steps of a call in one launch.
//
// The reciprocal sum of a step needs every charge's new position and the v / a
// update needs its forces, so with separate kernels a step was three dependent
// launches, and the lane kernel began each with a cold instruction cache, a
// load of the lane, its lists expanded and its near lists recorded anew: 62 us
// a step for 51 nucleotides with ions (lane 40, structure factors 8, forces 8
// us), 43 us for 21.  Here the launch is cooperative and its last CTAs are
// workers for the reciprocal sum, beside the lanes' clusters:
//   lane    e^{i 2 pi x / L} of its charges at the new positions -> ready
//           (then its own sweep, while the workers sum)
//   workers S(k) of a column (hx, hy) per 128 threads -> barrier of the
//           workers -> forces, a thread per column -> done
//   lane    waits for done at the end of its sweep
// EWF_NOW.  The powers of a charge's exponentials replace the columns' sincos.
// A worker's 512 threads have 128 registers, so a column's 12 hz are two
// halves there; with 256 threads the whole column.
//
// Counters only grow during a launch (zeroed before it).  Every wait is
// bounded: one that gives up raises the abort flag, with which all waits
// return at once, so every CTA still takes all its steps and ends; the lanes
// are flagged (LF_WAIT).
#pragma once
#include "device_common.cuh"

namespace tis {

constexpr int EW_WAIT_POLLS = 4000000;   // about 2 s
constexpr int EW_WQ = 8;                 // charges of a worker's force block at most

__device__ __forceinline__ void ew_wait(const KArgs &a, int word, unsigned target) {
  for (int i = 0;; ++i) {
    unsigned v, ab;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a.ew_sync + word) : "memory");
    if ((int)(v - target) >= 0) return;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(ab) : "l"(a.ew_sync + EWS_ABORT) : "memory");
    if (ab) return;
    if (i == EW_WAIT_POLLS) {
      atomicExch(a.ew_sync + EWS_ABORT, 1u);
      return;
    }
  }
}

// called by one thread after a barrier behind the writes it announces
__device__ __forceinline__ void ew_signal(const KArgs &a, int word) {
  __threadfence();
  atomicAdd(a.ew_sync + word, 1u);
}

__device__ __forceinline__ double2 cmul(double2 x, double2 y) {
  return make_double2(fma(x.x, y.x, -(x.y * y.y)), fma(x.x, y.y, x.y * y.x));
}

// z^n, 0 <= n < 16
__device__ __forceinline__ double2 cpow(double2 z, int n) {
  double2 r = make_double2(1.0, 0.0);
#pragma unroll 1
  for (; n; n >>= 1) {
    if (n & 1) r = cmul(r, z);
    z = cmul(z, z);
  }
  return r;
}

template <int NT>
__device__ __forceinline__ void ewald_worker(const KArgs &a, unsigned char *smem) {
  constexpr int HV = NT >= 512 ? 2 : 1, HN = EW_H / HV, G = NT / 128, NWRP = NT / 32;
  const int tid = threadIdx.x, lid = tid & 31, warp = tid >> 5;
  const int nw = a.ew_nwork, w = (int)(blockIdx.x - (gridDim.x - nw));
  const int ncol = a.ew_ncol, CP = (ncol + 31) & ~31, nqm = a.ew_nqmax;
  double *red = (double *)smem;                              // [G][4][4 HN]
  double2 *ex = (double2 *)(red + G * 16 * HN);              // [EW_WQ][3][EW_H]
  double *rf = (double *)(ex + EW_WQ * 3 * EW_H);            // [NWRP][EW_WQ][3]
  const int per = min(EW_WQ, (nqm * a.nlane + nw - 1) / nw), blocks = (nqm + per - 1) / per;
  for (int step = 0; step < a.nsteps; ++step) {
    if (tid == 0) ew_wait(a, EWS_READY, (unsigned)(step + 1) * (unsigned)(a.nlane * a.nsplit));
    __syncthreads();
    // ---- structure factors, see ewald_kernel.cu: 128 threads a column (or half of one)
    {
      const int g = tid >> 7, t = tid & 127;
      double *r4 = red + g * 16 * HN;
      for (int u = w + nw * g; u < a.nlane * ncol * HV; u += nw * G) {
        const int lane = u / (ncol * HV), cu = u - lane * (ncol * HV), c = cu / HV, h0 = (cu - c * HV) * HN;
        const char4 col = a.ew_col[c];
        const int mz = col.z, hx = col.x, hy = abs(col.y);
        if (h0 > mz) continue;   // the same for the whole group
        const LaneDesc L = a.lanes[lane];
        const TopDesc T = a.tops[L.top];
        const double2 *E = a.ew_E + (size_t)lane * 3 * nqm;
        double P[HN], Q[HN], R[HN], U[HN];
#pragma unroll
        for (int h = 0; h < HN; ++h) P[h] = Q[h] = R[h] = U[h] = 0.0;
        for (int k = t; k < T.nq; k += 128) {
          const double q = a.b_charge[T.bead0 + a.q_bead[T.q0 + k]];
          const double2 x = cpow(__ldcg(E + k), hx), z = __ldcg(E + 2 * nqm + k);
          double2 y = cpow(__ldcg(E + nqm + k), hy);
          if (col.y < 0) y.y = -y.y;
          const double2 v = cmul(x, y);
          const double ca = q * v.x, cb = q * v.y;
          double2 e = cpow(z, h0);
#pragma unroll
          for (int h = 0; h < HN; ++h) {
            if (h0 + h > mz) break;
            if (h || HV > 1) {
              P[h] = fma(ca, e.x, P[h]); Q[h] = fma(cb, e.y, Q[h]); R[h] = fma(ca, e.y, R[h]); U[h] = fma(cb, e.x, U[h]);
            } else {
              P[h] += ca; U[h] += cb;
            }
            e = cmul(e, z);
          }
        }
#pragma unroll
        for (int h = 0; h < HN; ++h) {
          if (h0 + h > mz) break;
          double v[4] = {P[h], Q[h], R[h], U[h]};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
            if (lid == 0) r4[(warp & 3) * 4 * HN + 4 * h + q] = v[q];
          }
        }
        asm volatile("bar.sync %0, 128;" ::"r"(1 + g) : "memory");
        if (t < 4 * HN && h0 + (t >> 2) <= mz) {
          double v = 0.0;
          for (int q = 0; q < 4; ++q) v += r4[q * 4 * HN + t];
          a.ew_S[(((size_t)lane * EW_H + h0 + (t >> 2)) * ncol + c) * 4 + (t & 3)] = v;
        }
        asm volatile("bar.sync %0, 128;" ::"r"(1 + g) : "memory");
      }
    }
    __syncthreads();
    if (tid == 0) {
      ew_signal(a, EWS_BARRIER);
      ew_wait(a, EWS_BARRIER, (unsigned)(step + 1) * (unsigned)nw);
    }
    __syncthreads();
    // ---- forces of `per` charges: a thread per column (or half of one)
    for (int u = w; u < a.nlane * blocks; u += nw) {
      const int lane = u / blocks, k0 = (u - lane * blocks) * per;
      const LaneDesc L = a.lanes[lane];
      const TopDesc T = a.tops[L.top];
      const int nk = min(per, T.nq - k0);
      if (nk <= 0) continue;   // the same for the whole CTA
      const double2 *E = a.ew_E + (size_t)lane * 3 * nqm;
      for (int e = tid; e < nk * 3 * EW_H; e += NT) {
        const int q = e / (3 * EW_H), d = (e / EW_H) % 3, h = e % EW_H;
        if (h <= a.hmax) ex[e] = cpow(__ldcg(E + d * nqm + k0 + q), h);
      }
      const int hv = tid >= CP ? 1 : 0, c = tid - hv * CP, h0 = hv * HN;
      const bool on = c < ncol && hv < HV;
      const char4 col = on ? a.ew_col[c] : make_char4(0, 0, -1, 0);
      const int mz = col.z, mw = __reduce_max_sync(0xffffffffu, mz);   // CP is a multiple of 32: h0 is the warp's
      double p[HN], r[HN], s[HN], t[HN];
#pragma unroll
      for (int h = 0; h < HN; ++h) {
        p[h] = r[h] = s[h] = t[h] = 0.0;
        if (h0 + h <= mz) {
          const double2 *S = (const double2 *)(a.ew_S + (((size_t)lane * EW_H + h0 + h) * ncol + c) * 4);
          const double2 S0 = __ldcg(S), S1 = __ldcg(S + 1);
          const double wt = a.ew_w[(h0 + h) * ncol + c];
          p[h] = wt * S0.x; s[h] = -(wt * S0.y); t[h] = wt * S1.x; r[h] = wt * S1.y;
        }
      }
      __syncthreads();
      if (h0 <= mw)
        for (int q = 0; q < nk; ++q) {
          const double2 *eq = ex + q * 3 * EW_H;
          const double2 vx = eq[col.x];
          double2 vy = eq[EW_H + abs(col.y)];
          if (col.y < 0) vy.y = -vy.y;
          const double2 cab = cmul(vx, vy);
          double g1 = 0.0, g2 = 0.0, h1 = 0.0, h2 = 0.0;
#pragma unroll
          for (int h = 0; h < HN; ++h) {
            if (h0 + h > mw) break;   // the warp's longest column (sums beyond a column's own are zero)
            const double2 z = eq[2 * EW_H + h0 + h];
            const double fh = (double)(h0 + h), ch = fh * z.x, dh = fh * z.y;
            g1 = fma(z.x, p[h], fma(z.y, t[h], g1));
            g2 = fma(z.y, s[h], fma(-z.x, r[h], g2));
            h1 = fma(ch, s[h], fma(dh, r[h], h1));
            h2 = fma(dh, p[h], fma(-ch, t[h], h2));
          }
          const double dv = fma(cab.y, g1, cab.x * g2), dz = fma(cab.y, h1, cab.x * h2);
          double f[3] = {dv * (double)col.x, dv * (double)col.y, dz};
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            for (int o = 16; o > 0; o >>= 1) f[d] += __shfl_xor_sync(0xffffffffu, f[d], o);
            if (lid == 0) rf[(warp * EW_WQ + q) * 3 + d] = f[d];
          }
        }
      else if (lid < 3 * nk)
        rf[warp * EW_WQ * 3 + lid] = 0.0;
      __syncthreads();
      if (tid < 3 * nk) {
        const int q = tid / 3, d = tid - 3 * q;
        const int bead = a.q_bead[T.q0 + k0 + q];
        double f = 0.0;
        for (int v = 0; v < NWRP; ++v) f += rf[(v * EW_WQ + q) * 3 + d];
        // force_ele_coulomb_ewld.F90:74-80 (see ewald_kernel.cu)
        const double coef = 4.0 * a.lab_coef[a.lstate[lane].label] * a.b_charge[T.bead0 + bead] * a.two_pi_L;
        a.f_ext[3 * (size_t)(L.state0 + bead) + d] = coef * f;
      }
      __syncthreads();
    }
    __syncthreads();
    if (tid == 0) ew_signal(a, EWS_DONE);
  }
}

} // namespace tis
