// ewald_kernel.cu -- reciprocal-space Ewald sums on the device, FP64
// (force_ele_coulomb_ewld.F90:62-84 forces, energy_ele_coulomb_ewld.F90:75-89
// energy, k vectors of mloop_ewld.F90:56-156).
//
// For a charge at x, e^{i k.x} with k = 2 pi (hx, hy, hz) / L factorises
// into e^{i 2 pi hx x / L} e^{i 2 pi hy y / L} e^{i 2 pi hz z / L} = (a + i b)
// (c + i d), with (c, d) of -hz the conjugate of hz's.  The vectors are taken
// by columns (hx, hy) of the half space hx > 0, or hx = 0 and hy >= 0 (-k adds
// the same force and energy as k, so sums over it are doubled; the column
// (0, 0) holds both k and -k and weighs half).  For the pair +-hz of a column
// the four sums over the charges
//   P = sum q a c   Q = sum q b d   R = sum q a d   T = sum q b c
// give both structure factors, S(+-hz) = (P -+ Q) + i (T +- R): four products
// a charge for two vectors, and as many for their force on a charge.
//
//   ewald_sk_kernel     one block per column: threads over the charges, the
//                       column's sums in registers, one reduction at the end
//   ewald_force_kernel  one block per few charges: a thread per column keeps
//                       its sums, weighted, in registers for all of them
//   ewald_energy_kernel per lane: coef (sum_k C(k) |S(k)|^2 + self)
//
// A table of the charges' exponentials, structure factors per block of 64
// charges with a kernel that adds them, and forces by k range of one vector
// at a time took 8.9 + 14.6 + 5.4 + 19.5 us for 641 charges and 4,168 vectors
// (four launches; 8.8 + 9.8 + 3.2 + 12.7 us for 165 charges): ten times the
// FP64 work of the column form and four dependent launches.
//
// Steps of lanes split over clusters take these sums inside their own launch
// where enough CTAs are left (split_ewald.cuh: 62 -> 20 us a step for 51
// nucleotides with 590 ions); these kernels serve single-point calls, one-CTA
// lanes, batches that fill the chip and replicas with their own step counts.
//
// All sums run in a fixed order, so the results do not depend on scheduling.
#include <algorithm>

#include "device_common.cuh"

namespace tis {

constexpr int EW_SK_THREADS = 128;
constexpr int EW_F_MAXQ = 8;   // charges of a force block at most

// grid (columns, lanes): S[(lane 12 + h) ncol + col] = (P, Q, R, T) of +-h
__global__ void __launch_bounds__(EW_SK_THREADS) ewald_sk_kernel(KArgs a) {
  const int lane = (a.only_lane >= 0) ? a.only_lane : (int)blockIdx.y;
  if (lane >= a.nlane) return;
  const LaneDesc L = a.lanes[lane];
  const TopDesc T = a.tops[L.top];
  const char4 col = a.ew_col[blockIdx.x];   // hx, hy, largest hz
  const double hx = (double)col.x * a.two_pi_L, hy = (double)col.y * a.two_pi_L;
  const int mz = col.z;
  double P[EW_H], Q[EW_H], R[EW_H], U[EW_H];
#pragma unroll
  for (int h = 0; h < EW_H; ++h) P[h] = Q[h] = R[h] = U[h] = 0.0;
  for (int k = threadIdx.x; k < T.nq; k += EW_SK_THREADS) {
    const int bead = a.q_bead[T.q0 + k];
    const double *x = a.pxyz + 3 * (size_t)(L.state0 + bead);
    const double q = a.b_charge[T.bead0 + bead];
    double sx, cx, sy, cy, s1, c1;
    sincos(hx * x[0], &sx, &cx);
    sincos(hy * x[1], &sy, &cy);
    sincos(a.two_pi_L * x[2], &s1, &c1);
    const double ca = q * (cx * cy - sx * sy), cb = q * (cx * sy + sx * cy);
    P[0] += ca; U[0] += cb;
    double c = c1, d = s1;
#pragma unroll
    for (int h = 1; h < EW_H; ++h) {
      if (h > mz) break;
      P[h] = fma(ca, c, P[h]); Q[h] = fma(cb, d, Q[h]); R[h] = fma(ca, d, R[h]); U[h] = fma(cb, c, U[h]);
      const double c2 = c * c1 - d * s1;   // e^{i (h + 1) z}
      d = fma(c, s1, d * c1);
      c = c2;
    }
  }
  constexpr int NWRP = EW_SK_THREADS / 32;
  __shared__ double red[NWRP][4 * EW_H];
  const int lid = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int h = 0; h < EW_H; ++h) {
    if (h > mz) break;
    double v[4] = {P[h], Q[h], R[h], U[h]};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
      if (lid == 0) red[warp][4 * h + q] = v[q];
    }
  }
  __syncthreads();
  if (threadIdx.x < 4 * (mz + 1)) {
    double v = 0.0;
    for (int w = 0; w < NWRP; ++w) v += red[w][threadIdx.x];
    a.ew_S[(((size_t)lane * EW_H + (threadIdx.x >> 2)) * a.ew_ncol + blockIdx.x) * 4 + (threadIdx.x & 3)] = v;
  }
}

// grid (ceil(nq / per), lanes), one thread per column (rounded up to whole
// warps): the forces of `per` charges
__global__ void __launch_bounds__(EW_COLS) ewald_force_kernel(KArgs a, int per) {
  const int lane = (a.only_lane >= 0) ? a.only_lane : (int)blockIdx.y;
  if (lane >= a.nlane) return;
  const LaneDesc L = a.lanes[lane];
  const TopDesc T = a.tops[L.top];
  const int k0 = blockIdx.x * per, nk = min(per, T.nq - k0);
  if (nk <= 0) return;
  const int tid = threadIdx.x, lid = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  __shared__ double2 ex[EW_F_MAXQ][3][EW_H];   // (cos, sin)(2 pi h x_d / L) of the block's charges
  __shared__ double red[EW_COLS / 32][EW_F_MAXQ][3];
  for (int e = tid; e < nk * 3 * EW_H; e += blockDim.x) {
    const int q = e / (3 * EW_H), d = (e / EW_H) % 3, h = e % EW_H;
    if (h <= a.hmax) {
      const double x = a.pxyz[3 * (size_t)(L.state0 + a.q_bead[T.q0 + k0 + q]) + d];
      double sn, cs;
      sincos((double)h * (a.two_pi_L * x), &sn, &cs);
      ex[q][d][h] = make_double2(cs, sn);
    }
  }
  // this column's weighted sums
  const bool on = tid < a.ew_ncol;
  const char4 col = on ? a.ew_col[tid] : make_char4(0, 0, -1, 0);
  const int mz = col.z, mw = __reduce_max_sync(0xffffffffu, mz);
  double p[EW_H], r[EW_H], s[EW_H], t[EW_H];
#pragma unroll
  for (int h = 0; h < EW_H; ++h) {
    p[h] = r[h] = s[h] = t[h] = 0.0;
    if (h <= mz) {
      const double *S = a.ew_S + (((size_t)lane * EW_H + h) * a.ew_ncol + tid) * 4;
      const double w = a.ew_w[h * a.ew_ncol + tid];
      p[h] = w * S[0]; s[h] = -(w * S[1]); t[h] = w * S[2]; r[h] = w * S[3];
    }
  }
  __syncthreads();
  for (int q = 0; q < nk; ++q) {
    const double2 vx = ex[q][0][col.x], vy0 = ex[q][1][abs(col.y)];
    const double sy = col.y < 0 ? -vy0.y : vy0.y;
    const double ca = vx.x * vy0.x - vx.y * sy, cb = fma(vx.x, sy, vx.y * vy0.x);
    double g1 = p[0], g2 = -r[0], h1 = 0.0, h2 = 0.0;
#pragma unroll
    for (int h = 1; h < EW_H; ++h) {
      if (h > mw) break;   // the warp's longest column (sums beyond a column's own are zero)
      const double2 z = ex[q][2][h];
      const double c = z.x, d = z.y, ch = (double)h * c, dh = (double)h * d;
      g1 = fma(c, p[h], fma(d, t[h], g1));
      g2 = fma(d, s[h], fma(-c, r[h], g2));
      h1 = fma(ch, s[h], fma(dh, r[h], h1));
      h2 = fma(dh, p[h], fma(-ch, t[h], h2));
    }
    const double dv = fma(cb, g1, ca * g2), dz = fma(cb, h1, ca * h2);
    double f[3] = {dv * (double)col.x, dv * (double)col.y, dz};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      for (int o = 16; o > 0; o >>= 1) f[d] += __shfl_xor_sync(0xffffffffu, f[d], o);
      if (lid == 0) red[warp][q][d] = f[d];
    }
  }
  __syncthreads();
  if (tid < 3 * nk) {
    const int q = tid / 3, d = tid - 3 * q;
    const int bead = a.q_bead[T.q0 + k0 + q];
    double f = 0.0;
    for (int w = 0; w < nw; ++w) f += red[w][q][d];
    // dv of a vector: coef 2 C(k) q (sin S_c - cos S_s) (force_ele_coulomb_ewld.F90:74-80), twice for -k
    const double coef = 4.0 * a.lab_coef[a.lstate[lane].label] * a.b_charge[T.bead0 + bead] * a.two_pi_L;
    a.f_ext[3 * (size_t)(L.state0 + bead) + d] = coef * f;
  }
}

// grid nlane, 256 threads: adds coef (E_f + E_s) to E_ELE and E_TOTAL of each
// lane's energy (energy_ele_coulomb_ewld.F90:75-89 and the self term :212)
__global__ void __launch_bounds__(256) ewald_energy_kernel(KArgs a) {
  const int lane = (a.only_lane >= 0) ? a.only_lane : (int)blockIdx.x;
  if (lane >= a.nlane) return;
  const LaneDesc L = a.lanes[lane];
  const TopDesc T = a.tops[L.top];
  const int label = (a.elabel && a.elabel[lane] >= 0) ? a.elabel[lane] : a.lstate[lane].label;
  double ef = 0.0, qq = 0.0;
  for (int k = threadIdx.x; k < EW_H * a.ew_ncol; k += blockDim.x) {
    const int h = k / a.ew_ncol, col = k - h * a.ew_ncol;
    if (h > a.ew_col[col].z) continue;
    const double *S = a.ew_S + ((size_t)lane * EW_H * a.ew_ncol + k) * 4;
    ef += 2.0 * a.ew_w[k] * ((S[0] * S[0] + S[1] * S[1]) + (S[2] * S[2] + S[3] * S[3]));
  }
  for (int kq = threadIdx.x; kq < T.nq; kq += blockDim.x) {
    const double q = a.b_charge[T.bead0 + a.q_bead[T.q0 + kq]];
    qq += q * q;
  }
  __shared__ double red[2][8];
  for (int o = 16; o > 0; o >>= 1) {
    ef += __shfl_xor_sync(0xffffffffu, ef, o);
    qq += __shfl_xor_sync(0xffffffffu, qq, o);
  }
  if ((threadIdx.x & 31) == 0) { red[0][threadIdx.x >> 5] = ef; red[1][threadIdx.x >> 5] = qq; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double e = 0.0, s = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) { e += red[0][w]; s += red[1][w]; }
    const double add = a.lab_coef[label] * (e + a.ewld_self * s);
    double *E = a.out_energy + (size_t)lane * N_ETYPE;
    E[7] += add;
    E[0] += add;
  }
}

// Launches structure factors and forces (into f_ext) for one lane
// (only_lane >= 0) or every lane.  nq_max: largest charge count of a lane.
cudaError_t ewald_recip_launch(cudaStream_t st, const KArgs &a, int nq_max, bool forces) {
  if (forces && !a.f_ext) return cudaErrorInvalidValue;
  const int nl = a.only_lane >= 0 ? 1 : a.nlane;
  ewald_sk_kernel<<<dim3(a.ew_ncol, nl), EW_SK_THREADS, 0, st>>>(a);
  if (forces && nq_max > 0) {
    // as few charges a block as still fill the chip once
    const int per = std::min(EW_F_MAXQ, std::max(1, (int)(((long long)nq_max * nl + 147) / 148)));
    ewald_force_kernel<<<dim3((nq_max + per - 1) / per, nl), (a.ew_ncol + 31) / 32 * 32, 0, st>>>(a, per);
  }
  return cudaGetLastError();
}

cudaError_t ewald_energy_launch(cudaStream_t st, const KArgs &a) {
  ewald_energy_kernel<<<a.only_lane >= 0 ? 1 : a.nlane, 256, 0, st>>>(a);
  return cudaGetLastError();
}

} // namespace tis
