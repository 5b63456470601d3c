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
//   lane    powers of e^{i 2 pi x / L} of its beads at the new positions -> ready
//           (then its own sweep, while the workers sum)
//   workers S(k) of a column (hx, hy) per 128 threads -> barrier of the
//           workers -> forces, a thread per column -> done
//   lane    waits for done at the end of its sweep
// 20 us a step for 51 nucleotides with 590 ions, 19 for 21 with 144 (FP64): the
// workers' chain of structure factors 8 k cycles, barrier 2.5 k, forces 8 to 11 k
// hides the lanes' sweep (7 to 10 k), and update, publication and the two
// signals (14 k) hide from the workers.  The published powers of a charge's
// exponentials replace the columns' sincos.
// A worker's 512 threads have 128 registers, so a column's 12 hz are two
// halves there; with 256 threads the whole column.
//
// Counters only grow during a launch (zeroed before it).  Every wait is
// bounded: one that gives up raises the abort flag, with which all waits
// return at once, so every CTA still takes all its steps and ends; the lanes
// are flagged (LF_WAIT).
#pragma once
#include "device_common.cuh"
#include "split_plan.cuh"

namespace tis {

// By a whole warp: after a loop that one thread takes alone the warp stayed in
// two parts, up to the next shuffle (4 k cycles of a lane's update).
__device__ __forceinline__ void ew_wait(const KArgs &a, int word, unsigned target) {
  const unsigned *p = a.ew_sync + word;
  for (int i = 0;; ++i) {
    unsigned v, ab;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    if ((int)(v - target) >= 0) break;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(ab) : "l"(a.ew_sync + EWS_ABORT) : "memory");
    if (ab) break;
    if (i >= a.ew_polls) {
      asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a.ew_sync + EWS_ARRIVED) : "memory");
      if (v >= gridDim.x || i >= EW_START_WAIT * a.ew_polls) {
        atomicExch(a.ew_sync + EWS_ABORT, 1u);
        break;
      }
    }
  }
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  __syncwarp();
}

// called by one thread after a barrier behind the writes it announces
__device__ __forceinline__ void ew_signal(const KArgs &a, int word) {
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.ew_sync + word) : "memory");
}

__device__ __forceinline__ double2 cmul(double2 x, double2 y) {
  return make_double2(fma(x.x, y.x, -(x.y * y.y)), fma(x.x, y.y, x.y * y.x));
}

// Own beads' powers e^{i 2 pi h x_d / L}, h = 0 .. hmax, for the workers:
// ew_E[(h 3 + d) nb + bead], nb beads of the context; P: wrapped coordinates,
// component stride np, beads lo ..
__device__ __forceinline__ void ew_publish(const KArgs &a, const double *P, int np, int lo, int nown, int state0,
                                           int tid, int nt) {
  for (int q = tid; q < 3 * nown; q += nt) {
    const int d = q / nown, i = lo + q - d * nown;
    double2 z, v = make_double2(1.0, 0.0);
    sincos(a.two_pi_L * P[d * np + i], &z.y, &z.x);
    double2 *E = a.ew_E + (size_t)d * a.ew_nb + state0 + i;
    for (int h = 0; h <= a.hmax; ++h) {
      __stcg(E, v);
      E += 3 * (size_t)a.ew_nb;
      v = cmul(v, z);
    }
  }
}

// sums over a warp of 32 values per lane, lane l receiving value l: each of
// five exchanges halves the values (31 shuffles instead of 5 per value)
template <int NV>
__device__ __forceinline__ double reduce_scatter(double (&v)[NV], int lid) {
#pragma unroll
  for (int o = 16, n = NV / 2; o; o >>= 1, n >>= 1) {
    if (n) {
#pragma unroll
      for (int i = 0; i < NV / 2; ++i)
        if (i < n) {
          const bool up = lid & o;
          const double keep = up ? v[i + n] : v[i], give = up ? v[i] : v[i + n];
          v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    }
  }
  return v[0];   // value lid / (32 / NV)
}

template <int NT>
__device__ __forceinline__ void ewald_worker(const KArgs &a, unsigned char *smem) {
  constexpr int HV = NT >= 512 ? 2 : 1, HN = EW_H / HV, G = NT / 128, NWRP = NT / 32;
  const int tid = threadIdx.x, lid = tid & 31, warp = tid >> 5;
  const int nw = a.ew_nwork, w = (int)(blockIdx.x - (gridDim.x - nw));
  const int ncol = a.ew_ncol, CP = (ncol + 31) & ~31, nqm = a.ew_nqmax;
  const size_t nb = a.ew_nb, hs = 3 * nb;   // rows of ew_E: a component, a power
  const EwSmem m = ew_smem(a.nlane, nqm, ncol);
  double *red = (double *)(smem + m.red);                    // [G][4][4 HN]
  double2 *ex = (double2 *)(smem + m.ex);                    // [EW_WQ][3][EW_H]
  double *rf = (double *)(smem + m.rf);                      // [NWRP][32]
  double *wt = (double *)(smem + m.wt), *bq = (double *)(smem + m.bq);
  int *bi = (int *)(smem + m.bi);
  double2 *ln = (double2 *)(smem + m.lane);                  // (factor, charges)
  char4 *cols = (char4 *)(smem + m.col);
  for (int k = tid; k < EW_H * ncol; k += NT) wt[k] = a.ew_w[k];
  for (int k = tid; k < ncol; k += NT) cols[k] = a.ew_col[k];
  for (int l = warp; l < a.nlane; l += NWRP) {
    const LaneDesc L = a.lanes[l];
    const TopDesc T = a.tops[L.top];
    for (int k = lid; k < T.nq; k += 32) {
      const int bead = a.q_bead[T.q0 + k];
      bi[l * nqm + k] = L.state0 + bead;
      bq[l * nqm + k] = a.b_charge[T.bead0 + bead];
    }
    // force_ele_coulomb_ewld.F90:74-80 (see ewald_kernel.cu)
    if (lid == 0) ln[l] = make_double2(4.0 * a.lab_coef[a.lstate[l].label] * a.two_pi_L, (double)T.nq);
  }
  __syncthreads();
  const int per = min(EW_WQ, (nqm * a.nlane + nw - 1) / nw), blocks = (nqm + per - 1) / per;
  for (int step = 0; step < a.nsteps; ++step) {
    if (warp == 0) ew_wait(a, EWS_READY, (unsigned)(step + 1) * (unsigned)(a.nlane * a.nsplit));
    __syncthreads();
    // ---- structure factors, see ewald_kernel.cu: 128 threads a column (or half of one)
    {
      const int g = tid >> 7, t = tid & 127;
      double *r4 = red + g * 16 * HN;
      for (int u = w + nw * g; u < a.nlane * ncol * HV; u += nw * G) {
        const int lane = u / (ncol * HV), cu = u - lane * (ncol * HV), c = cu / HV, h0 = (cu - c * HV) * HN;
        const char4 col = cols[c];
        const int mz = col.z;
        if (h0 > mz) continue;   // the same for the whole group
        const double2 *Ex = a.ew_E + col.x * hs, *Ey = a.ew_E + abs(col.y) * hs + nb, *Ez = a.ew_E + 2 * nb;
        const int nq = (int)ln[lane].y, *b = bi + lane * nqm;
        const double *qv = bq + lane * nqm;
        double S[32 * ((HN + 7) / 8)];   // P, Q, R, T of h0 + h at 4 h
#pragma unroll
        for (int k = 0; k < 32 * ((HN + 7) / 8); ++k) S[k] = 0.0;
        double2 x, y, z, e;
        auto fetch = [&](int k) {
          if (k < nq) {
            const int at = b[k];
            x = __ldcg(Ex + at);
            y = __ldcg(Ey + at);
            z = __ldcg(Ez + hs + at);
            e = __ldcg(Ez + h0 * hs + at);
          }
        };
        fetch(t);
        for (int k = t; k < nq; k += 128) {
          if (col.y < 0) y.y = -y.y;
          const double2 v = cmul(x, y), z1 = z;
          const double q = qv[k], ca = q * v.x, cb = q * v.y;
          double2 eh = e;
          fetch(k + 128);
#pragma unroll
          for (int h = 0; h < HN; ++h) {
            if (h0 + h > mz) break;
            S[4 * h] = fma(ca, eh.x, S[4 * h]);
            S[4 * h + 1] = fma(cb, eh.y, S[4 * h + 1]);
            S[4 * h + 2] = fma(ca, eh.y, S[4 * h + 2]);
            S[4 * h + 3] = fma(cb, eh.x, S[4 * h + 3]);
            eh = cmul(eh, z1);
          }
        }
#pragma unroll
        for (int p = 0; p < (HN + 7) / 8; ++p) {
          double v[32];
#pragma unroll
          for (int k = 0; k < 32; ++k) v[k] = S[32 * p + k];
          const double r = reduce_scatter<32>(v, lid);
          if (32 * p + lid < 4 * HN) r4[(warp & 3) * 4 * HN + 32 * p + lid] = r;
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
    if (tid == 0) ew_signal(a, EWS_BARRIER);
    if (warp == 0) ew_wait(a, EWS_BARRIER, (unsigned)(step + 1) * (unsigned)nw);
    __syncthreads();
    // ---- forces of `per` charges: a thread per column (or half of one)
    for (int u = w; u < a.nlane * blocks; u += nw) {
      const int lane = u / blocks, k0 = (u - lane * blocks) * per;
      const int nk = min(per, (int)ln[lane].y - k0), *b = bi + lane * nqm + k0;
      if (nk <= 0) continue;   // the same for the whole CTA
      for (int e = tid; e < nk * 3 * EW_H; e += NT) {
        const int q = e / (3 * EW_H), d = (e / EW_H) % 3, h = e % EW_H;
        if (h <= a.hmax) ex[e] = __ldcg(a.ew_E + h * hs + d * nb + b[q]);
      }
      const int hv = tid >= CP ? 1 : 0, c = tid - hv * CP, h0 = hv * HN;
      const bool on = c < ncol && hv < HV;
      const char4 col = on ? cols[c] : make_char4(0, 0, -1, 0);
      const int mz = col.z, mw = __reduce_max_sync(0xffffffffu, mz);   // CP is a multiple of 32: h0 is the warp's
      double p[HN], r[HN], s[HN], t[HN];
#pragma unroll
      for (int h = 0; h < HN; ++h) {   // all loads in flight: a column without this h reads its first one
        const bool ok = h0 + h <= mz;
        const int at = (ok ? h0 + h : 0) * ncol + (on ? c : 0);
        const double2 *S = (const double2 *)(a.ew_S + ((size_t)lane * EW_H * ncol + at) * 4);
        const double2 S0 = __ldcg(S), S1 = __ldcg(S + 1);
        const double f = wt[at];
        p[h] = ok ? f * S0.x : 0.0; s[h] = ok ? -(f * S0.y) : 0.0;
        t[h] = ok ? f * S1.x : 0.0; r[h] = ok ? f * S1.y : 0.0;
      }
      __syncthreads();
      if (h0 <= mw)
#pragma unroll 1
        for (int q0 = 0; q0 < nk; q0 += 4) {
          double f[16];   // charge q0 + q, component d at 4 q + d
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const double2 *eq = ex + min(q0 + q, nk - 1) * 3 * EW_H;
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
            f[4 * q] = dv * (double)col.x;
            f[4 * q + 1] = dv * (double)col.y;
            f[4 * q + 2] = dz;
            f[4 * q + 3] = 0.0;
          }
          const double v = reduce_scatter<16>(f, lid);   // lanes 2 k, 2 k + 1: value k
          if (!(lid & 1)) rf[warp * 32 + 4 * q0 + (lid >> 1)] = v;
        }
      else
        rf[warp * 32 + lid] = 0.0;
      __syncthreads();
      if (tid < 32 && (tid & 3) < 3 && (tid >> 2) < nk) {
        double f = 0.0;
        for (int v = 0; v < NWRP; ++v) f += rf[v * 32 + tid];
        a.f_ext[3 * (size_t)b[tid >> 2] + (tid & 3)] = ln[lane].x * bq[lane * nqm + k0 + (tid >> 2)] * f;
      }
      __syncthreads();
    }
    __syncthreads();
    if (tid == 0) ew_signal(a, EWS_DONE);
  }
}

} // namespace tis
