// split_plan.cuh -- shared-memory layout of a lane split over a cluster
// (split_kernel.cuh), shared with the host, which lays out the constant part.
#pragma once
#include "common.cuh"

namespace tis {

constexpr int SG = 8;            // threads per bead (update phase, exv lists)
constexpr int SP_NEAR = 8;       // near-list entries per thread of a bead's group
// near lists: partners within the screen radius + SP_SKIN, recorded by every
// CTA of a lane together as soon as any bead has moved SP_SKIN_DISP since (two
// beads then close in by less than SP_SKIN - 0.1 A).  A wider skin than the
// one-CTA kernel's: a recording scans the exv rows (~8 k cycles for 1,199
// beads on 16 CTAs), a list entry out of reach costs one screened pair
constexpr float SP_SKIN = 2.0f;
constexpr float SP_SKIN_DISP = 0.95f;
constexpr int SP_IMG = 11;       // pair entries: bead in the low bits, periodic image above (periodic lanes: N < 2048)

// threads of a warp that share one charged row: short rows take few
__host__ __device__ inline int split_row_lanes(int nq, bool ewald) {
  return (ewald || nq <= 64) ? 8 : (nq <= 160 ? 16 : 32);
}

// own beads of a CTA for a lane of N beads
__host__ __device__ inline int split_own(int N, int nr) { return ((N + nr - 1) / nr + 3) & ~3; }

// threads of a CTA: 256 (with twice the registers) while its warps have a few
// work items each, 512 above
inline int split_threads(int N, int nr) { return split_own(N, nr) <= 32 ? 256 : 512; }

// T: the largest counts of the context's topologies; bonded items: of a CTA
// row: partners of a charged row to make room for (on average over a CTA's rows)
inline SplitPlan split_plan(const TopDesc &T, int nq, int row, int nr, bool periodic, bool skin, bool ewald, int real,
                            unsigned limit) {
  SplitPlan p;
  const int N = T.nmp;
  p.own = split_own(N, nr);
  p.rows = (nq + nr - 1) / nr;
  p.nst = T.nst; p.nhb = T.nhb; p.nba = T.nba; p.nbd = T.nbd; p.nts = T.ntst;
  p.np = (N + 3) & ~3;
  const unsigned n = p.np, o = p.own, W = (N + 31) / 32, R = real;
  unsigned b = 0;
  auto take = [&](unsigned bytes) { const unsigned at = b; b = (b + bytes + 15u) & ~15u; return at; };
  p.tcu = take(4 * n);                    // type | class << 4 | unit << 8 (and the kernel's periodic cell << 16)
  p.RE = take(2 * R * n);                 // exv radius, sqrt(eps)
  p.qb = take(4 * nq);
  p.base = take(4 * (SPLIT_MAX + 1));
  p.rn2 = take(8 * T.nunit * T.nunit);
  p.comm = b;
  p.C = take(32 * o);                     // rlan_const(2..4), 1 / m of the own beads
  p.scr = take(R * o);                    // exv screen radius
  p.iptr = take(4 * (o + 1));
  p.cnt = take(4 * 5);                    // hydrogen bonds, stacks, tertiary stacks, angles, bonds of the CTA
  p.stk = take(4 * p.nst); p.hbk = take(4 * p.nhb); p.tsk = take(4 * p.nts);   // their numbers in the topology
  p.bdi = take(4 * p.nbd); p.bdd = take(8 * p.nbd); p.bdc = take(2 * R * p.nbd);
  p.bai = take(8 * p.nba); p.bad = take(12 * p.nba); p.bac = take(2 * R * p.nba);
  p.sti = take(16 * p.nst); p.std_ = take(28 * p.nst); p.stc = take(6 * R * p.nst);
  p.hbi = take(12 * p.nhb); p.hbd = take(24 * p.nhb); p.hbc = take(13 * R * p.nhb); p.hbs = take(24 * p.nhb);
  p.stat = b;
  p.X = take(24 * n);
  p.P = periodic ? take(24 * n) : p.X;
  p.Q = periodic ? take(24 * n) : p.X;
  p.A4 = take(4 * R * (n + 4));           // and a bead far away without charge (entry np)
  p.L3 = real == 4 ? take(12 * n) : 0;
  p.V = take((skin ? 72 : 48) * o);       // v, a, [dxyz]
  p.DD = skin ? take(8 * o) : 0;
  p.C1 = take(8 * o);
  p.u0 = take(8 * p.nst);
  p.NZ = take(24 * o); p.exF = take(24 * o); p.dhF = take(24 * o);
  p.NR4 = take(16 * o);
  p.near = take(2 * SG * SP_NEAR * o); p.ncnt = take(SG * o);
  p.mexv = take(4 * W * o); p.mele = take(4 * W * p.rows);
  p.slots = take(3 * R * T.sp_ninc);
  p.exc = take(4 * T.nsite); p.hbf = take(p.nhb);
  p.red = take(8 * (64 + 2 * SPLIT_MAX) + 16 * SPLIT_MAX);   // reductions; then the CTAs' displacement maxima, 2 parities
  p.img = periodic ? take(4 * R * 27) : 0;
  p.misc = take(4 * (SPLIT_MISC + T.nunit * T.nunit + 8));
  // partner lists of the charged rows, or what is left of the shared memory
  const unsigned eb = 2 * split_row_lanes(nq, ewald), most = p.rows * (((row < nq ? row : nq) + eb - 1) / eb * eb);
  p.eoff = take(4 * (p.rows + 1));
  const unsigned left = b < limit ? (limit - b) / 32 * 16 : 0;
  p.ecap = most < left ? most : left;
  p.elist = take(2 * p.ecap);
  p.total = b;
  return p;
}

// Workers of the reciprocal Ewald sum (split_ewald.cuh).
constexpr int EW_WQ = 8;   // charges of a force block at most
// Their shared memory: reductions, the force block's exponentials, and
// what never changes during a launch (the waits drop L1, so it would come from
// L2 step after step, through four dependent loads)
struct EwSmem {
  unsigned red, ex, rf, wt, bq, bi, lane, col, total;
};
__host__ __device__ inline EwSmem ew_smem(int nlane, int nqm, int ncol) {
  EwSmem m;
  unsigned b = 0;
  auto take = [&](unsigned bytes) { const unsigned at = b; b = (b + bytes + 15u) & ~15u; return at; };
  m.red = take(8 * 4 * 16 * 6);                // sums of the warps: 512 threads 4 groups x 24, 256 threads 2 x 48
  m.ex = take(16 * EW_WQ * 3 * EW_H);
  m.rf = take(8 * 16 * 32);
  m.wt = take(8 * EW_H * ncol);
  m.bq = take(8 * nlane * nqm);                // charges, in the order of
  m.bi = take(4 * nlane * nqm);                // their rows in ew_E
  m.lane = take(16 * nlane);                   // force factor, charges
  m.col = take(4 * ncol);
  m.total = b;
  return m;
}

} // namespace tis
