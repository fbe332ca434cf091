// kernels_fp64.cuh -- FP64 kernels of the lapw1 H/S setup (sm_100a).
//
// Data layout in HBM for one k-point (rows = HSROWS = nv + nlo, padded):
//   al, bl     [nat][ltop][nvpad]  f64    matching coefficients (K-a)
//   phase      [ndf][npad]         c128   exp(2 pi i K_n . r_a) of every row
//   tab        [(2d3+1)(2d2+1)(2d1+1)] 2 x c128: (Theta(dK), WARP(dK))
//   hns L / R  [ndf*2*nsl2][npad]  c128   HNS left (A2,B2) / right (ALM,BLM)
//   hs         n x n c128, column-major (the caller's HS), hsdiag n c128
#pragma once
#include "common.cuh"

struct DevProb {
  int n, nv, nlo, nat, ndf, ltop, ldl, lnsmax, ins;
  int nvpad, npad;
  double vi;
  // structure
  const int* mult;
  const int* atype;     // [ndf] 0-based type of atom a
  const int* afirst;    // [nat] first atom index of type
  const double* rmt;
  const double* v;
  const double* pos;    // [ndf][3]
  const double* rotij;  // [ndf][9]
  const double* rotloc; // [nat][9]
  // rows
  const int* kzz;       // [n][3]
  const double* xk;
  const double* yk;
  const double* zk;
  const double* rk;
  // radial [nat][ldl]
  const double* p;
  const double* pe;
  const double* dp;
  const double* dpe;
  const double* pei;
  const double* e;
  const int* lapw;
  // LO
  const int* ilo;
  const int* loor;
  const double* alo;
  const double* blo;
  const double* clo;
  const double* elo;
  const double* pi12lo;
  const double* pe12lo;
  const double* dplo;
  // derived
  double* al;
  double* bl;
  double2* phase;
};

// ---------------------------------------------------------------------
// K-a: AL/BL (hamilt.F:160-175), one thread per (row n < nv, atom type)
// ---------------------------------------------------------------------
__global__ void k_albl(DevProb P, int* status) {
  int n = blockIdx.x * blockDim.x + threadIdx.x;
  int jn = blockIdx.y;
  if (n >= P.nvpad) return;
  const int ltop = P.ltop;
  double* al = P.al + ((size_t)jn * ltop) * P.nvpad + n;
  double* bl = P.bl + ((size_t)jn * ltop) * P.nvpad + n;
  if (n >= P.nv) {
    for (int l = 0; l < ltop; l++) {
      al[(size_t)l * P.nvpad] = 0.0;
      bl[(size_t)l * P.nvpad] = 0.0;
    }
    return;
  }
  double fj[L1G_MAXL + 2], dfj[L1G_MAXL + 2];
  double rkn = P.rk[n], r = P.rmt[jn];
  int st = dev_sphbes(ltop - 1, r * rkn, fj);
  if (st) atomicOr(status, st);
  dev_dvbes1(fj, dfj, rkn, r, ltop);
  const double* U = P.p + jn * P.ldl;
  const double* UP = P.pe + jn * P.ldl;
  const double* DU = P.dp + jn * P.ldl;
  const double* DUP = P.dpe + jn * P.ldl;
  const int* LAPW = P.lapw + jn * P.ldl;
  for (int l = 0; l < ltop; l++) {
    double a, b;
    if (LAPW[l]) {
      a = rkn * dfj[l] * UP[l] - fj[l] * DUP[l];
      b = fj[l] * DU[l] - rkn * dfj[l] * U[l];
    } else {
      a = fj[l] / U[l] / (r * r);
      b = 0.0;
    }
    al[(size_t)l * P.nvpad] = a;
    bl[(size_t)l * P.nvpad] = b;
  }
}

// structure-factor phases of every row for every atom (hns.F:171-174)
__global__ void k_phase(DevProb P) {
  int n = blockIdx.x * blockDim.x + threadIdx.x;
  int a = blockIdx.y;
  if (n >= P.npad) return;
  double2 v = cmk(0.0, 0.0);
  if (n < P.n) {
    const double* r = P.pos + 3 * a;
    const int* k = P.kzz + 3 * n;
    double s = r[0] * (double)k[0] + r[1] * (double)k[1] + r[2] * (double)k[2];
    v = cexp2pi(s);
  }
  P.phase[(size_t)a * P.npad + n] = v;
}

// ---------------------------------------------------------------------
// K-c table: Theta(dK) and WARP(dK) on the integer box of row differences.
//   INS == 0: Theta(dK != 0) = sum_type 3 V PHASE BESR  (hamilt.F:297-326)
//             Theta(0)       = sum_type (1/NAT - V MULT) (hamilt.F:328-329)
//   INS != 0: USTPHX (ustphx.F:31-52); no warp term (hamilt.F:349-365)
// ---------------------------------------------------------------------
struct TabDesc {
  int d1, d2, d3;       // half extents
  int w1, w2, w3;       // WARP half extents
  double bk[9];         // Cartesian dK = bk * dKZZ  (bk row-major [3][3])
};

__global__ void k_table(DevProb P, TabDesc T, const double2* warp, double2* tab) {
  int nx = 2 * T.d1 + 1, ny = 2 * T.d2 + 1, nz = 2 * T.d3 + 1;
  int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= nx * ny * nz) return;
  int ix = idx % nx, iy = (idx / nx) % ny, iz = idx / (nx * ny);
  int d[3] = {ix - T.d1, iy - T.d2, iz - T.d3};
  double g0 = T.bk[0] * d[0] + T.bk[1] * d[1] + T.bk[2] * d[2];
  double g1 = T.bk[3] * d[0] + T.bk[4] * d[1] + T.bk[5] * d[2];
  double g2 = T.bk[6] * d[0] + T.bk[7] * d[1] + T.bk[8] * d[2];
  double slen = sqrt(g0 * g0 + g1 * g1 + g2 * g2);
  bool zero = (d[0] == 0 && d[1] == 0 && d[2] == 0);
  double2 th = cmk(0.0, 0.0);
  if (P.ins == 0) {
    for (int jn = 0; jn < P.nat; jn++) {
      if (zero) {
        th.x = th.x + 1.0 / (double)P.nat - P.v[jn] * (double)P.mult[jn];
      } else {
        double2 ph = cmk(0.0, 0.0);
        int a0 = P.afirst[jn];
        for (int q = 0; q < P.mult[jn]; q++) {
          const double* r = P.pos + 3 * (a0 + q);
          ph = cadd(ph, cexp2pi(r[0] * d[0] + r[1] * d[1] + r[2] * d[2]));
        }
        double h = slen * P.rmt[jn];
        double sn, cs;
        sincos(h, &sn, &cs);
        double besr = (h * cs - sn) * (1.0 / (h * h * h));
        double v3 = 3.0 * P.v[jn];
        th = cadd(th, cscale(cscale(ph, v3), besr));
      }
    }
  } else {
    if (slen > 1.0e-10) {
      double2 u = cmk(0.0, 0.0);
      for (int jn = 0; jn < P.nat; jn++) {
        double2 ph = cmk(0.0, 0.0);
        int a0 = P.afirst[jn];
        for (int q = 0; q < P.mult[jn]; q++) {
          const double* r = P.pos + 3 * (a0 + q);
          ph = cadd(ph, cexp2pi(r[0] * d[0] + r[1] * d[1] + r[2] * d[2]));
        }
        double qq = slen * P.rmt[jn];
        double sn, cs;
        sincos(qq, &sn, &cs);
        double besr = (qq * cs - sn) / (qq * qq * qq);
        u = cadd(u, cscale(cscale(ph, P.v[jn]), besr));
      }
      th = cscale(u, 3.0);
    } else {
      double u = 0.0;
      for (int jn = 0; jn < P.nat; jn++) u = u + P.v[jn] * (double)P.mult[jn];
      th = cmk(1.0 - u, 0.0);
    }
  }
  double2 w = cmk(0.0, 0.0);
  if (P.ins == 0 && abs(d[0]) <= T.w1 && abs(d[1]) <= T.w2 && abs(d[2]) <= T.w3) {
    size_t wi = ((size_t)(d[2] + T.w3) * (2 * T.w2 + 1) + (size_t)(d[1] + T.w2)) * (2 * T.w1 + 1) +
                (size_t)(d[0] + T.w1);
    w = warp[wi];
  }
  tab[2 * (size_t)idx] = th;
  tab[2 * (size_t)idx + 1] = w;
}

// ---------------------------------------------------------------------
// K-b + K-c: PW x PW block of H and S (hamilt.F:188-466 + ZSWAP).
//
// Per pair (J <= I), the reference accumulates, atom type by atom type,
//   t_S = sum_l (2l+1) P_l(x_JI) [AL_J AL_I + CHN BL_J BL_I]
//   t_H = sum_l (2l+1) P_l(x_JI) [AL_J hA_I + BL_J hB_I]
// with hA/hB the non-symmetric 2x2 block of hamilt.F:386-424 (surface
// kinetic terms included) applied on the column side, and adds
// VIF * PHASE * t to S and H, PHASE = sum_eq exp(2 pi i (K_J - K_I) r_eq).
// This kernel keeps that loop order: the Legendre weights w_l = (2l+1) P_l
// of each pair are computed once with the reference's recursion (UTOP
// branch included, hamilt.F:250-281) and held in registers; per atom type
// the J-side {AL, BL} and the I-side VIF {AL, CHN BL, hA, hB} rows
// (k_pair_rows) are staged in shared memory; PHASE is formed as
// sum_eq phi_a(J) conj(phi_a(I)) from the per-row phases.  That is 6 FP64
// operations per (pair, type, l) plus the phase products, instead of 16 for
// the same sum as a GEMM over explicit (l, r).
// ---------------------------------------------------------------------
#define SPH_T 32
#define SPH_THREADS 256
#define SPH_LMAX 13

struct SphCoef {  // per (type, l)
  double vif, chn, mAA, mAB, mBA, mBB;
};

__global__ void k_sph_coef(DevProb P, SphCoef* coef) {
  int l = threadIdx.x, jn = blockIdx.x;
  if (l >= P.ltop) return;
  const double pi = 3.141592653589793238462643;
  double r = P.rmt[jn];
  double r2 = r * r;
  int o = jn * P.ldl + l;
  double U = P.p[o], UP = P.pe[o], DU = P.dp[o], DUP = P.dpe[o], CHN = P.pei[o], E = P.e[o];
  SphCoef c;
  c.vif = 4.0 * pi * P.vi * (r2 * r2);
  c.chn = P.lapw[o] ? CHN : 0.0;
  c.mAA = E + r2 * (U * DU);
  c.mAB = r2 * (UP * DU);
  c.mBA = 1.0 + r2 * (U * DUP);
  c.mBB = E * CHN + r2 * (UP * DUP);
  coef[jn * P.ltop + l] = c;
}

// Operand rows of the pair kernels (k_spherical, k_force_sph), per (type, l, row): the J side
// (a, b) and the I side, S = vif (a, chn b) and H = vif (mAA a + mAB b,
// mBA a + mBB b), so that each l term of a pair is one 2-vector dot
// product per side.  Rows nv..nvpad-1 are zero (k_albl zeroes them).
__global__ void k_pair_rows(DevProb P, const SphCoef* __restrict__ coef, double2* __restrict__ rowJ,
                             double2* __restrict__ rowI) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x, tl = blockIdx.y;  // tl = type * ltop + l
  if (r >= P.nvpad) return;
  const size_t o = (size_t)tl * P.nvpad + r;
  const double a = P.al[o], b = P.bl[o];
  const SphCoef c = coef[tl];
  rowJ[o] = cmk(a, b);
  rowI[2 * o] = cmk(c.vif * a, c.vif * (c.chn * b));
  rowI[2 * o + 1] = cmk(c.vif * (c.mAA * a + c.mAB * b), c.vif * (c.mBA * a + c.mBB * b));
}

// Rows of a lane in the pair kernels: J row (0..7) and I row (0..3).  A 128-bit
// shared load takes two cycles where lanes i and i ^ 1 (I rows) or i and i ^ 2
// (J rows) of each half warp read one address, and four otherwise.  With J =
// lane & 7, I = lane >> 3 the J loads took four: 2.5 per load on the mean against
// 1.9 now, k_spherical 3.48 -> 3.37 ms and k_force_sph 3.90 -> 3.77 (40 atoms, nv 4600).
__device__ __forceinline__ int pr_lane_j(int lane) { return (lane & 1) | ((lane >> 1) & 6); }
__device__ __forceinline__ int pr_lane_i(int lane) { return ((lane >> 1) & 1) | ((lane >> 3) & 2); }

#define PR_MAXA 16  // equivalent atoms per staged chunk (a type with more reads its phases from global)
#define PR_LT 11    // l count of the specialised kernel (lmax = 10)

// types per staged chunk: as many as the shared memory holds twice
__host__ __device__ constexpr int pr_tc(int lt) { return lt <= PR_LT ? 5 : 4; }

// 16-byte global -> shared copy that bypasses registers (cp.async), so that
// a block's staging has all its loads in flight at once
__device__ __forceinline__ void pr_cp16(void* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void pr_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void pr_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// A chunk of types from t0: up to TC types whose equivalent atoms fit
// PR_MAXA; a single type with more atoms forms a chunk of its own whose
// phases are not staged.
struct PairChunk {
  int ntc, na, staged;
};
template <int TC>
__device__ __forceinline__ PairChunk pr_chunk(const DevProb& P, int t0) {
  PairChunk c{0, 0, 1};
  while (c.ntc < TC && t0 + c.ntc < P.nat && c.na + P.mult[t0 + c.ntc] <= PR_MAXA) c.na += P.mult[t0 + c.ntc++];
  if (c.ntc == 0) c = PairChunk{1, 0, 0};
  return c;
}

// dynamic shared memory of k_spherical: two stages of type rows (J: 1, I: 2
// double2 per row and l) and of phases
__host__ __device__ constexpr int sph_smem_bytes(int lt) {
  return (2 * pr_tc(lt) * lt * SPH_T * 3 + 2 * 2 * PR_MAXA * SPH_T) * 16;
}

// One block per 32 x 32 pair tile, 256 threads, bound by the FP64 pipe's
// issue.  Thread (warp, lane) owns the 2 x 2 pairs J = j0 + jl0 + {0, 8},
// I = i0 + il0 + {0, 4} with jl0 = 16 (warp & 1) + pr_lane_j, il0 =
// 8 (warp >> 1) + pr_lane_i: a warp reads 8 distinct J rows and 4 distinct
// I rows per l, 6 shared loads of two cycles for 24 FP64 operations.  (2 x 1
// pairs in 16 warps: 4 loads for 12, 4.5% slower; 12 warps of 2 x 2: spills.)  The chunk of types after the current one is
// copied by cp.async meanwhile (one block barrier per chunk), and for
// one-atom types the phase products of a type are formed beside the l sums
// of the next.  LT: l values (unrolled); GUARD: ltop may be below LT.
template <int LT, bool GUARD>
__global__ void __launch_bounds__(SPH_THREADS, 1)
    k_spherical(DevProb P, const int2* __restrict__ tiles, const double2* __restrict__ rowJ,
                const double2* __restrict__ rowI, const double2* __restrict__ tab, TabDesc T, double2* __restrict__ hs,
                int ld, double2* __restrict__ hsdiag, int* __restrict__ status) {
  constexpr int TC = pr_tc(LT);
  extern __shared__ double2 sm2[];
  double2* sJ = sm2;                       // [2][TC][LT][SPH_T]
  double2* sI = sJ + 2 * TC * LT * SPH_T;  // [2][TC][LT][SPH_T][S, H]
  double2* sP = sI + 4 * TC * LT * SPH_T;  // [2][J, I][PR_MAXA][SPH_T]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int2 t = tiles[blockIdx.x];
  const int i0 = t.x * SPH_T, j0 = t.y * SPH_T;
  const int nv = P.nv, ltop = P.ltop, nat = P.nat, nvpad = P.nvpad;
  const int jl0 = (warp & 1) * 16 + pr_lane_j(lane), il0 = (warp >> 1) * 8 + pr_lane_i(lane);

  // (type, l) rows of consecutive types are consecutive in rowJ / rowI
  auto stage = [&](int st, int t0, const PairChunk& ch) {
    double2* dJ = sJ + st * TC * LT * SPH_T;
    double2* dI = sI + st * 2 * TC * LT * SPH_T;
    const size_t g0 = (size_t)t0 * ltop;
    for (int k = warp; k < ch.ntc * ltop; k += SPH_THREADS / 32) {
      const int ks = GUARD ? (k / ltop) * LT + k % ltop : k;
      const double2* src = rowJ + (g0 + k) * nvpad + j0;
      pr_cp16(dJ + ks * SPH_T + lane, src + lane);
      const double2* srci = rowI + 2 * ((g0 + k) * nvpad + i0);
      pr_cp16(dI + ks * 2 * SPH_T + lane, srci + lane);
      pr_cp16(dI + ks * 2 * SPH_T + SPH_T + lane, srci + SPH_T + lane);
    }
    if (ch.staged) {
      double2* dP = sP + st * 2 * PR_MAXA * SPH_T;
      const int a0c = P.afirst[t0];
      for (int k = warp; k < ch.na * 2; k += SPH_THREADS / 32) {
        const int side = k & 1, e = k >> 1;
        pr_cp16(dP + (side * PR_MAXA + e) * SPH_T + lane,
                P.phase + (size_t)(a0c + e) * P.npad + (side ? i0 : j0) + lane);
      }
    }
    pr_commit();
  };
  PairChunk ch = pr_chunk<TC>(P, 0);
  stage(0, 0, ch);

  // Legendre weights (2l+1) P_l(x_JI) of the four owned pairs
  double w[4][LT];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int J = j0 + jl0 + 8 * (q >> 1), I = i0 + il0 + 4 * (q & 1);
    double x = 0.0;
    if (J < nv && I < nv) {
      x = P.xk[I] * P.xk[J] + P.yk[I] * P.yk[J] + P.zk[I] * P.zk[J];
      const double den = P.rk[I] * P.rk[J];
      if (den > 1.0e-8) x = x / den;
    }
    const bool top = !(fabs(x) < 0.9999999);
    double pm2 = 1.0, pm1 = x;
    w[q][0] = 1.0;
    if (LT > 1) w[q][1] = 3.0 * x;
#pragma unroll
    for (int l = 2; l < LT; l++) {
      double pl;
      if (!top) {
        const double pplx = x * pm1;
        pl = pplx + ((double)(l - 1) / (double)l) * (pplx - pm2);
      } else {
        pl = x * pm1;
      }
      pm2 = pm1;
      pm1 = pl;
      w[q][l] = (double)(2 * l + 1) * pl;
    }
  }
  double2 aS[4], aH[4];
#pragma unroll
  for (int q = 0; q < 4; q++) aS[q] = aH[q] = cmk(0.0, 0.0);

  int st = 0;
  for (int t0 = 0; t0 < nat;) {
    const int t1 = t0 + ch.ntc;
    pr_wait<0>();
    __syncthreads();  // every thread's copies landed; every warp is past the previous chunk
    PairChunk nx{0, 0, 1};
    if (t1 < nat) {  // into the stage the previous chunk read
      nx = pr_chunk<TC>(P, t1);
      stage(st ^ 1, t1, nx);
    }
    const double2* cJ = sJ + st * TC * LT * SPH_T + jl0;
    const double2* cI = sI + st * 2 * TC * LT * SPH_T + 2 * il0;
    const double2* cPJ = sP + st * 2 * PR_MAXA * SPH_T + jl0;
    const double2* cPI = sP + st * 2 * PR_MAXA * SPH_T + PR_MAXA * SPH_T + il0;
    // l sums of type tc for the four pairs (the row values of l + 1 are read
    // while l is summed)
    auto lsum = [&](int tc, double(&tS)[4], double(&tH)[4]) {
      const double2* bJ = cJ + tc * LT * SPH_T;
      const double2* bI = cI + tc * LT * 2 * SPH_T;
      double2 av[2] = {bJ[0], bJ[8]}, sv[2] = {bI[0], bI[8]}, hv[2] = {bI[1], bI[9]};
#pragma unroll
      for (int l = 0; l < LT; l++) {
        if (GUARD && l >= ltop) break;
        const double2 a0 = av[0], a1 = av[1], s0 = sv[0], s1 = sv[1], h0 = hv[0], h1 = hv[1];
        if (l + 1 < LT) {
          const int o = (l + 1) * SPH_T;
          av[0] = bJ[o];
          av[1] = bJ[o + 8];
          sv[0] = bI[2 * o];
          sv[1] = bI[2 * o + 8];
          hv[0] = bI[2 * o + 1];
          hv[1] = bI[2 * o + 9];
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const double2 a = (q >> 1) ? a1 : a0, s = (q & 1) ? s1 : s0, h = (q & 1) ? h1 : h0;
          if (l == 0) {  // w_0 = P_0 = 1
            tS[q] = fma(a.y, s.y, a.x * s.x);
            tH[q] = fma(a.y, h.y, a.x * h.x);
          } else {
            tS[q] = fma(w[q][l], fma(a.y, s.y, a.x * s.x), tS[q]);
            tH[q] = fma(w[q][l], fma(a.y, h.y, a.x * h.x), tH[q]);
          }
        }
      }
    };
    // phi_J conj(phi_I) of one atom added to ph
    auto phase = [&](const double2(&fj)[2], const double2(&fi)[2], double2(&ph)[4]) {
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const double2 a = fj[q >> 1], b = fi[q & 1];
        ph[q].x = fma(a.x, b.x, fma(a.y, b.y, ph[q].x));
        ph[q].y = fma(a.y, b.x, fma(-a.x, b.y, ph[q].y));
      }
    };
    auto add = [&](const double2(&ph)[4], const double(&tS)[4], const double(&tH)[4]) {
#pragma unroll
      for (int q = 0; q < 4; q++) {
        aS[q].x = fma(ph[q].x, tS[q], aS[q].x);
        aS[q].y = fma(ph[q].y, tS[q], aS[q].y);
        aH[q].x = fma(ph[q].x, tH[q], aH[q].x);
        aH[q].y = fma(ph[q].y, tH[q], aH[q].y);
      }
    };
    auto one = [&](int e, const double(&tS)[4], const double(&tH)[4]) {  // a one-atom type, staged slot e
      const double2 fj[2] = {cPJ[e * SPH_T], cPJ[e * SPH_T + 8]}, fi[2] = {cPI[e * SPH_T], cPI[e * SPH_T + 4]};
      double2 ph[4] = {};
      phase(fj, fi, ph);
      add(ph, tS, tH);
    };
    if (ch.staged && ch.na == ch.ntc) {
      double pS[4], pH[4];
      lsum(0, pS, pH);
      for (int tc = 1; tc < ch.ntc; tc++) {
        double tS[4], tH[4];
        lsum(tc, tS, tH);
        one(tc - 1, pS, pH);
#pragma unroll
        for (int q = 0; q < 4; q++) {
          pS[q] = tS[q];
          pH[q] = tH[q];
        }
      }
      one(ch.ntc - 1, pS, pH);
    } else {
      const int a0c = P.afirst[t0];
      for (int tc = 0; tc < ch.ntc; tc++) {
        double tS[4], tH[4];
        lsum(tc, tS, tH);
        const int jn = t0 + tc, ae = P.afirst[jn], me = P.mult[jn];
        double2 ph[4] = {};
        for (int e = 0; e < me; e++) {
          double2 fj[2], fi[2];
          if (ch.staged) {
            const int b = (ae - a0c + e) * SPH_T;
            fj[0] = cPJ[b];
            fj[1] = cPJ[b + 8];
            fi[0] = cPI[b];
            fi[1] = cPI[b + 4];
          } else {  // a type with more atoms than a chunk stages
            const double2* pa = P.phase + (size_t)(ae + e) * P.npad;
            fj[0] = pa[j0 + jl0];
            fj[1] = pa[j0 + jl0 + 8];
            fi[0] = pa[i0 + il0];
            fi[1] = pa[i0 + il0 + 4];
          }
          phase(fj, fi, ph);
        }
        add(ph, tS, tH);
      }
    }
    t0 = t1;
    ch = nx;
    st ^= 1;
  }
  // interstitial + write (hamilt.F:289-345, 459-466, calkpt.F:164); a non-finite
  // written element sets L1G_STATUS_NONFINITE
  const int nx = 2 * T.d1 + 1, ny = 2 * T.d2 + 1;
  bool bad = false;
#pragma unroll
  for (int v = 0; v < 2; v++) {
    const int I = i0 + il0 + 4 * v;
    if (I >= nv) continue;
    const int k1 = P.kzz[3 * I], k2 = P.kzz[3 * I + 1], k3 = P.kzz[3 * I + 2];
    const double xi = P.xk[I], yi = P.yk[I], zi = P.zk[I];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const int J = j0 + jl0 + 8 * u;
      if (J > I) continue;
      const int q = u * 2 + v;
      const double x2 = P.xk[J] * xi + P.yk[J] * yi + P.zk[J] * zi;
      const int d1 = P.kzz[3 * J] - k1 + T.d1, d2 = P.kzz[3 * J + 1] - k2 + T.d2, d3 = P.kzz[3 * J + 2] - k3 + T.d3;
      const size_t c = ((size_t)d3 * ny + d2) * nx + d1;
      const double2 th = tab[2 * c], wp = tab[2 * c + 1];
      const double2 s = cadd(th, aS[q]);
      const double2 h = cadd(cadd(cscale(th, x2), wp), aH[q]);
      if (J == I) {
        hs[(size_t)I * ld + I] = h;
        hsdiag[I] = s;
      } else {
        hs[(size_t)I * ld + J] = s;  // S upper: HS(J,I)
        hs[(size_t)J * ld + I] = h;  // H lower: HS(I,J)
      }
      bad |= l1g_nonfinite(s) | l1g_nonfinite(h);
    }
  }
  if (bad) atomicOr(status, L1G_STATUS_NONFINITE);
}

// ---------------------------------------------------------------------
// K-b': local-orbital columns (hamilt.F:475-818).  For LO column I (type t, l,
// index jlo, atom jeqo, mo1) and row J the reference sums over the equivalent
// atoms and m products of i^l conj(Y_lm) of both rows with the radial factors;
// i^l cancels, and the radial factors depend on neither atom nor m, so
//   S, H (J,I) = (4 pi VI^(1/2) R^2)^2 {rs, rh} T,
//   T = sum_eq phi_a(J) conj(phi_a(I)) sum_m Y_lm(J) conj(Y_lm(I)).
// A block forms the 2l+1 columns (mo1) of one (t, l, jlo, jeqo) for 128 rows, so
// that a row's Y_lm, the dearest part, is formed once for all of them: 40
// atoms (N = 4937) 0.13 -> 0.065 ms, 100 atoms (N = 12677) 0.83 -> 0.38 against a
// block per column with every product formed per m.
// ---------------------------------------------------------------------
struct LoCol {
  int jn, l, jlo, jeqo, mo1, nnlo, a0;  // a0: first atom of the type
};
#define LO_YCH 8  // atoms whose Y_lm of the LO rows a block holds at a time

// radial factors of one LO column (all mo1 of a group share them)
struct LoRad {
  double p2;  // (4 pi VI^(1/2) R^2)^2
  double U, UP, c1, c2, c3, c11, c12, c13, akin;
};
__device__ __forceinline__ LoRad lo_radial(const DevProb& P, const LoCol& c) {
  const double pi = 3.141592653589793238462643;
  const int jn = c.jn, l = c.l, o = jn * P.ldl + l, lo4 = jn * (L1G_LOMAX + 1) + l;
  const int oo = (jn * L1G_NLOAT + c.jlo - 1) * (L1G_LOMAX + 1) + l;
  const double r = P.rmt[jn], pr = 4.0 * pi * sqrt(P.vi) * r * r;
  const double U = P.p[o], UP = P.pe[o], DU = P.dp[o], DUP = P.dpe[o], CHN = P.pei[o], E = P.e[o];
  const double A = P.alo[oo], B = P.blo[oo], Cc = P.clo[oo], ELO = P.elo[oo];
  const double PI12 = P.pi12lo[lo4], PE12 = P.pe12lo[lo4], DPL = P.dplo[lo4];
  LoRad q;
  q.p2 = pr * pr;
  q.U = U;
  q.UP = UP;
  q.c1 = A + PI12 * Cc;
  q.c2 = B * CHN + PE12 * Cc;
  q.c3 = Cc + PE12 * B + A * PI12;
  q.c11 = A * E + 0.5 * (B + Cc * PI12 * (ELO + E));
  q.c12 = B * CHN * E + 0.5 * (A + Cc * PI12 + Cc * PE12 * (ELO + E));
  q.c13 = Cc * ELO + 0.5 * (B * PI12 + (ELO + E) * (A * PI12 + PE12 * B));
  q.akin = 0.5 * r * r * (A * DU + B * DUP + Cc * DPL);
  return q;
}
// rs, rh of plane-wave row J < nv
__device__ __forceinline__ double2 lo_pw_factors(const DevProb& P, const LoCol& c, const LoRad& q, int J) {
  const size_t o = ((size_t)c.jn * P.ltop + c.l) * P.nvpad + J;
  const double al = P.al[o], bl = P.bl[o];
  return cmk(q.p2 * (al * q.c1 + bl * q.c2), q.p2 * (al * q.c11 + bl * q.c12 + (al * q.U + bl * q.UP) * q.akin));
}
// rs, rh of LO row J of the same type and l against column mo1 of the group
// (0, 0 outside the row ranges of hamilt.F:677-680, 1-based NNLO arithmetic)
__device__ __forceinline__ double2 lo_lo_factors(const DevProb& P, const LoCol& c, const LoRad& q, int J, int mo1) {
  const int l = c.l, mult = P.mult[c.jn], nnlo = c.nnlo + mo1 + l;
  double2 f = cmk(0.0, 0.0);
  for (int jlop = 1; jlop <= c.jlo; jlop++) {
    const int dj = c.jlo - jlop;
    const int jbeg = P.nv + nnlo - (mo1 + l) - (2 * l + 1) * (c.jeqo - 1) - dj * (2 * l + 1) * mult;
    const int jend = P.nv + nnlo - dj * (mo1 + l + 1) - dj * (c.jeqo - 1) * (2 * l + 1);
    if (J + 1 < jbeg || J + 1 > jend) continue;
    const int oo = (c.jn * L1G_NLOAT + jlop - 1) * (L1G_LOMAX + 1) + l;
    const double A = P.alo[oo], B = P.blo[oo], Cc = P.clo[oo];
    f.x += q.p2 * (A * q.c1 + B * q.c2 + Cc * q.c3);
    f.y += q.p2 * (A * q.c11 + B * q.c12 + Cc * q.c13);
  }
  return f;
}
// conj(Y_lm) of the group's LO rows for atoms e0 .. of the type, [row][atom][m]
__device__ __forceinline__ void lo_stage_y(const DevProb& P, const LoCol& c, int e0, double2 (*sy)[LO_YCH][7]) {
  const int nm = 2 * c.l + 1, ne = min(LO_YCH, P.mult[c.jn] - e0);
  for (int w = threadIdx.x; w < nm * ne; w += blockDim.x) {
    const int q = w / ne, e = w % ne, I = P.nv + c.nnlo - 1 + q, a = c.a0 + e0 + e;
    double2 y[16];
    dev_ylm_row<3>(P.xk[I], P.yk[I], P.zk[I], P.rotij + 9 * a, P.rotloc + 9 * c.jn, c.l, y);
    for (int m = 0; m < nm; m++) sy[q][e][m] = cconj(y[c.l * c.l + m]);
  }
}
// row J's Y_lm for atom a times its phase
__device__ __forceinline__ void lo_row_y(const DevProb& P, const LoCol& c, int J, int a, double2 (&v)[7]) {
  double2 y[16];
  dev_ylm_row<3>(P.xk[J], P.yk[J], P.zk[J], P.rotij + 9 * a, P.rotloc + 9 * c.jn, c.l, y);
  const double2 ph = P.phase[(size_t)a * P.npad + J];
#pragma unroll
  for (int m = 0; m < 7; m++) v[m] = m < 2 * c.l + 1 ? cmul(ph, y[min(c.l * c.l + m, 15)]) : cmk(0.0, 0.0);
}
// sum_m v_m conj(Y_lm(I)) conj(phi_a(I))
__device__ __forceinline__ double2 lo_dot(const DevProb& P, int nm, const double2 (&v)[7], const double2* sy, int I, int a) {
  double2 t = cmk(0.0, 0.0);
#pragma unroll
  for (int m = 0; m < 7; m++)
    if (m < nm) t = cadd(t, cmul(v[m], sy[m]));
  return cmul(t, cconj(P.phase[(size_t)a * P.npad + I]));
}

// cols[groups[y]]: the group's first column (mo1 = -l).  status: when non-null,
// a non-finite written element sets L1G_STATUS_NONFINITE.
__global__ void __launch_bounds__(128) k_lo(DevProb P, const LoCol* __restrict__ cols, const int* __restrict__ groups,
                                            double2* __restrict__ hs, int ld, double2* __restrict__ hsdiag,
                                            int* __restrict__ status) {
  __shared__ double2 sy[7][LO_YCH][7];
  const LoCol c = cols[groups[blockIdx.y]];
  const int nv = P.nv, nm = 2 * c.l + 1, I0 = nv + c.nnlo - 1, mult = P.mult[c.jn];
  const int J = blockIdx.x * blockDim.x + threadIdx.x;
  if ((int)(blockIdx.x * blockDim.x) > I0 + nm - 1) return;  // past the last column (block-uniform)
  const bool active = J < I0 + nm;
  const LoRad rad = lo_radial(P, c);
  double2 T[7];
#pragma unroll
  for (int q = 0; q < 7; q++) T[q] = cmk(0.0, 0.0);
  for (int e = 0; e < mult; e++) {
    if (e % LO_YCH == 0) {  // block-uniform
      __syncthreads();
      lo_stage_y(P, c, e, sy);
      __syncthreads();
    }
    if (!active) continue;
    double2 v[7];
    lo_row_y(P, c, J, c.a0 + e, v);
#pragma unroll
    for (int q = 0; q < 7; q++)
      if (q < nm) T[q] = cadd(T[q], lo_dot(P, nm, v, sy[q][e % LO_YCH], I0 + q, c.a0 + e));
  }
  if (!active) return;
  const double2 fpw = J < nv ? lo_pw_factors(P, c, rad, J) : cmk(0.0, 0.0);
  bool bad = false;
#pragma unroll
  for (int q = 0; q < 7; q++) {
    const int I = I0 + q;
    if (q >= nm || J > I) continue;
    const double2 f = J < nv ? fpw : lo_lo_factors(P, c, rad, J, q - c.l);
    const bool none = J >= nv && f.x == 0.0 && f.y == 0.0;
    const double2 S = none ? cmk(0.0, 0.0) : cscale(T[q], f.x), H = none ? cmk(0.0, 0.0) : cscale(T[q], f.y);
    if (J == I) {
      hs[(size_t)I * ld + I] = H;
      hsdiag[I] = S;
    } else {
      hs[(size_t)I * ld + J] = S;
      hs[(size_t)J * ld + I] = H;
    }
    bad |= l1g_nonfinite(S) | l1g_nonfinite(H);
  }
  if (status && bad) atomicOr(status, L1G_STATUS_NONFINITE);
}

// ---------------------------------------------------------------------
// K-ns operands (hns.F:165-437).  For atom a, k = (a*2 + r)*nsl2 + lm:
//   R[k][i] = {ALM, BLM}(i, lm)            (hns.F:190-259; r = 0, 1)
//   L[k][i] = {A2, B2}(i, lm)              (hns.F:381-434)
// with A2 = sum_b TUU conj(ALM) + TDU conj(BLM) + TUU21 conj(CLM), B2 the
// same with TUD, TDD, TUD21 (the TMP sums of hns.F:387-417: T times the
// conjugate).  CLM is non-zero only on the atom's own LO rows, so
//   k_hns_alm     builds R (and CLM, C-side of the LO rows) per row,
//   k_hns_tmul    forms L = M conj(R) per atom as a small complex GEMM,
//                 M = [[TUU, TDU], [TUD, TDD]] (2 nsl2 x 2 nsl2),
//   k_hns_lo_ops  adds the CLM terms of the LO rows and their C2.
// ---------------------------------------------------------------------
struct LoRange {
  int jn, l, jlo, i1, i2;  // rows nv+i1..nv+i2 (1-based LO indices)
};

__global__ void k_hns_alm(DevProb P, const LoRange* __restrict__ lor, int nlor, double2* __restrict__ Rop,
                          double2* __restrict__ Clo) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;  // row
  const int a = blockIdx.y;                              // atom
  const int nsl = P.lnsmax + 1, nsl2 = nsl * nsl;
  if (i >= P.npad) return;
  const size_t Kst = (size_t)P.npad;
  double2* RA = Rop + ((size_t)(a * 2 + 0) * nsl2) * Kst + i;
  double2* RB = Rop + ((size_t)(a * 2 + 1) * nsl2) * Kst + i;
  if (i >= P.n) {
    for (int lm = 0; lm < nsl2; lm++) RA[lm * Kst] = RB[lm * Kst] = cmk(0.0, 0.0);
    return;
  }
  const int jn = P.atype[a];
  const double pi = 3.141592653589793238462643;
  const double rhoatm = 4.0 * pi * sqrt(P.vi) * P.rmt[jn] * P.rmt[jn];
  const double2 ph = P.phase[(size_t)a * P.npad + i];
  double2 y[25];
  dev_ylm_row<4>(P.xk[i], P.yk[i], P.zk[i], P.rotij + 9 * a, P.rotloc + 9 * jn, nsl - 1, y);
  // LO identity of this row for this atom's type (hns.F:223-255, LOHNS)
  int myl = -1, myjlo = 0;
  if (i >= P.nv) {
    const int li = i - P.nv + 1;
    for (int q = 0; q < nlor; q++)
      if (lor[q].jn == jn && li >= lor[q].i1 && li <= lor[q].i2) {
        myl = lor[q].l;
        myjlo = lor[q].jlo;
      }
  }
  double2 cil = cmk(1.0, 0.0);
  int lm = 0;
  for (int l0 = 0; l0 < nsl; l0++) {
    for (int m0 = -l0; m0 <= l0; m0++, lm++) {
      const double2 tt = cmul(cmul(cil, ph), cconj(y[lm]));
      const double almr = rhoatm * tt.x, almi = rhoatm * tt.y;
      double2 A = cmk(0.0, 0.0), B = A, Cc = A;
      if (i < P.nv) {
        const size_t o = ((size_t)jn * P.ltop + l0) * P.nvpad + i;
        const double alv = P.al[o], blv = P.bl[o];
        B = cmk(blv * almr, blv * almi);
        A = cmk(alv * almr, alv * almi);
      } else if (l0 == myl) {
        const int oo = (jn * L1G_NLOAT + myjlo - 1) * (L1G_LOMAX + 1) + l0;
        B = cmk(P.blo[oo] * almr, P.blo[oo] * almi);
        Cc = cmk(P.clo[oo] * almr, P.clo[oo] * almi);
        A = cmk(P.alo[oo] * almr, P.alo[oo] * almi);
      }
      RA[lm * Kst] = A;
      RB[lm * Kst] = B;
      if (i >= P.nv) Clo[((size_t)a * nsl2 + lm) * (size_t)P.nlo + (i - P.nv)] = Cc;
    }
    cil = cmk(-cil.y, cil.x);
  }
}


// c += a b for one 8 x 8 tile and 4 k: lane holds a(lane / 4, lane % 4),
// b(lane % 4, lane / 4), c(lane / 4, 2 (lane % 4) + {0, 1})
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}
#define TMUL_I 64        // columns (basis rows i) per work item
#define TMUL_WARPS 4     // 16 columns each
#define TMUL_MF 7        // 8-row fragments: 56 >= 2 NSL2 = 50 rows
#define TMUL_KP 52       // k padded to whole steps of 4
#define TMUL_MS 52       // row strides in shared memory: the 8 lanes of a quarter-warp
#define TMUL_RS 66       // (4 k x 2 rows or columns) read 8 different 16-byte banks
#define TMUL_SMEM ((8 * TMUL_MF * TMUL_MS + TMUL_KP * TMUL_RS) * 16)
// L[(a, r_out, la)][i] = sum_{(r, b)} M[(r_out, la)][(r, b)] conj(R[(a, r, b)][i])
// on the FP64 tensor cores.  A work item is (atom, 64 columns i); block b
// takes the contiguous items [b per, (b+1) per) (one atom for most of them: M
// is staged again only when the atom changes).  A warp forms all rows of 16
// columns, 7 x 2 complex fragments; two blocks per SM, so that one stages while
// the other multiplies.  Measured: 40 atoms (N = 4937) 0.20 ms, 100 atoms (N =
// 12677) 1.19 ms, 25 GFLOP (20 accumulators per thread on the FMA pipe: 0.29 and
// 1.80).
__global__ void __launch_bounds__(32 * TMUL_WARPS, 2) k_hns_tmul(int npad, int nsl2, int ndf, int per,
                                                              const int* __restrict__ atype,
                                                              const double2* __restrict__ tns,
                                                              const double2* __restrict__ Rop,
                                                              double2* __restrict__ Lop) {
  extern __shared__ double2 tm[];
  const int K = 2 * nsl2;
  double2* sM = tm;                              // [8 MF][MS], zero beyond K x K
  double2* sR = tm + 8 * TMUL_MF * TMUL_MS;  // [KP][RS], zero beyond K
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int nch = (npad + TMUL_I - 1) / TMUL_I, nitem = nch * ndf;
  const int it0 = blockIdx.x * per, it1 = min(nitem, it0 + per);
  for (int idx = tid; idx < 8 * TMUL_MF * TMUL_MS + TMUL_KP * TMUL_RS; idx += 32 * TMUL_WARPS) tm[idx] = cmk(0.0, 0.0);
  int staged = -1;
  for (int item = it0; item < it1; item++) {
    const int a = item / nch, i0 = (item % nch) * TMUL_I;
    __syncthreads();  // the previous item's smem reads (or the zero fill) are done
    if (a != staged) {
      const double2* T = tns + (size_t)atype[a] * LAPW1GPU_NTNS * L1G_NSL2 * L1G_NSL2;
      for (int idx = tid; idx < K * K; idx += 32 * TMUL_WARPS) {
        const int row = idx / K, col = idx % K;
        const int ro = row / nsl2, la = row % nsl2, r = col / nsl2, b = col % nsl2;
        const int blk = ro == 0 ? (r == 0 ? 0 : 1) : (r == 0 ? 3 : 4);  // TUU TDU / TUD TDD
        pr_cp16(&sM[row * TMUL_MS + col], &T[((size_t)blk * L1G_NSL2 + la) * L1G_NSL2 + b]);
      }
      staged = a;
    }
    const double2* R = Rop + (size_t)a * K * npad;
    for (int idx = tid; idx < K * TMUL_I; idx += 32 * TMUL_WARPS) {
      const int k = idx / TMUL_I, c = idx % TMUL_I;  // npad is a multiple of 64
      pr_cp16(&sR[k * TMUL_RS + c], &R[(size_t)k * npad + i0 + c]);
    }
    pr_commit();
    pr_wait<0>();
    __syncthreads();
    double re[TMUL_MF][2][2], im[TMUL_MF][2][2];
#pragma unroll
    for (int u = 0; u < TMUL_MF; u++)
#pragma unroll
      for (int v = 0; v < 2; v++) re[u][v][0] = re[u][v][1] = im[u][v][0] = im[u][v][1] = 0.0;
    const double2* pM = sM + (lane >> 2) * TMUL_MS + (lane & 3);
    const double2* pR = sR + (lane & 3) * TMUL_RS + 16 * w + (lane >> 2);
    for (int k = 0; k < K; k += 4) {
      double2 m[TMUL_MF], x[2];
#pragma unroll
      for (int v = 0; v < 2; v++) x[v] = pR[k * TMUL_RS + 8 * v];
#pragma unroll
      for (int u = 0; u < TMUL_MF; u++) m[u] = pM[8 * u * TMUL_MS + k];
      // m conj(x)
#pragma unroll
      for (int u = 0; u < TMUL_MF; u++)
#pragma unroll
        for (int v = 0; v < 2; v++) {
          dmma(re[u][v], m[u].x, x[v].x);
          dmma(im[u][v], m[u].y, x[v].x);
        }
#pragma unroll
      for (int u = 0; u < TMUL_MF; u++)
#pragma unroll
        for (int v = 0; v < 2; v++) {
          dmma(re[u][v], m[u].y, x[v].y);
          dmma(im[u][v], -m[u].x, x[v].y);
        }
    }
    double2* L = Lop + (size_t)a * K * npad + i0 + 16 * w + 2 * (lane & 3);
#pragma unroll
    for (int u = 0; u < TMUL_MF; u++) {
      const int row = 8 * u + (lane >> 2);
      if (row < K)
#pragma unroll
        for (int v = 0; v < 2; v++)
#pragma unroll
          for (int e = 0; e < 2; e++) L[(size_t)row * npad + 8 * v + e] = cmk(re[u][v][e], im[u][v][e]);
    }
  }
}

// LO rows: A2 += TUU21 conj(CLM), B2 += TUD21 conj(CLM),
// C2 = TUU12 conj(ALM) + TDU12 conj(BLM) + TUU22 conj(CLM)  (hns.F:391-433).
// Block (32 la, 8) over 8 LO rows of an atom: a warp takes one of them, lane la.
// Bound by latency (the copy of the rows, then T per non-zero b, then L):
// with 32 rows per block, four in turn per warp, 27 us at six atoms, 12.7 now;
// 62 and 70 us at 100 atoms, where it runs beside the spherical stage.  A row has ALM, BLM, CLM on the atoms of its own type only, and
// there only at its own l: the sums run over the non-zero b (bits of a ballot;
// NaN counts as non-zero), 1 + 3 + 5 of 25 for s, p and d rows, and a row
// that is zero on the atom writes C2 = 0 and leaves L as it is.  A non-finite T
// entry that meets zeros only is reported all the same: with a zero it makes
// the full sums, and so HS, NaN.  The first block of each type looks.
#define LOOPS_ROWS 8
__global__ void __launch_bounds__(256) k_hns_lo_ops(DevProb P, const double2* __restrict__ tns,
                                                    double2* __restrict__ Lop, const double2* __restrict__ Rop,
                                                    const double2* __restrict__ Clo, double2* __restrict__ C2lo,
                                                    int* __restrict__ status) {
  __shared__ double2 sX[LOOPS_ROWS][3][L1G_NSL2];
  const int la = threadIdx.x, cy = threadIdx.y;
  const int c0 = blockIdx.x * LOOPS_ROWS;  // first LO row of the block
  const int a = blockIdx.y;
  const int nsl2 = (P.lnsmax + 1) * (P.lnsmax + 1);
  const size_t npad = P.npad;
  for (int q = threadIdx.y * 32 + threadIdx.x; q < LOOPS_ROWS * 3 * nsl2; q += 256) {
    const int r = q % LOOPS_ROWS, w = q / LOOPS_ROWS / nsl2, b = q / LOOPS_ROWS % nsl2;
    const int cc = c0 + r;
    double2 v = cmk(0.0, 0.0);
    if (cc < P.nlo) {
      const size_t i = P.nv + cc;
      if (w < 2)
        v = Rop[((size_t)(a * 2 + w) * nsl2 + b) * npad + i];
      else
        v = Clo[((size_t)a * nsl2 + b) * P.nlo + cc];
    }
    sX[r][w][b] = v;
  }
  if (blockIdx.x == 0 && a == P.afirst[P.atype[a]]) {
    const double2* Ta = tns + (size_t)P.atype[a] * LAPW1GPU_NTNS * L1G_NSL2 * L1G_NSL2;
    bool bad = false;
    for (int q = threadIdx.y * 32 + threadIdx.x; q < 5 * nsl2 * nsl2; q += 256) {
      const int w = q / (nsl2 * nsl2), lb = q % (nsl2 * nsl2);
      const int blk = w == 0 ? 2 : w + 4;  // TUU21; TUD21, TUU12, TDU12, TUU22
      bad |= l1g_nonfinite(__ldg(Ta + ((size_t)blk * L1G_NSL2 + lb / nsl2) * L1G_NSL2 + lb % nsl2));
    }
    if (bad) atomicOr(status, L1G_STATUS_NONFINITE);
  }
  __syncthreads();
  const double2* T = tns + (size_t)P.atype[a] * LAPW1GPU_NTNS * L1G_NSL2 * L1G_NSL2 + min(la, nsl2 - 1) * L1G_NSL2;
  const int r = cy, c = c0 + r;  // warp-uniform
  if (c < P.nlo) {
    bool nz = false;
    if (la < nsl2)
#pragma unroll
      for (int w = 0; w < 3; w++) nz |= sX[r][w][la].x != 0.0 || sX[r][w][la].y != 0.0;
    unsigned bits = __ballot_sync(0xffffffffu, nz);
    if (la >= nsl2) return;
    double2 da = cmk(0, 0), db = da, dc = da;
    const bool some = bits != 0;
    for (; bits; bits &= bits - 1) {
      const int b = __ffs(bits) - 1;
      const double2 A = cconj(sX[r][0][b]), B = cconj(sX[r][1][b]), Cc = cconj(sX[r][2][b]);
#define TT(blk) __ldg(T + (size_t)(blk)*L1G_NSL2 * L1G_NSL2 + b)
      const double2 tuu21 = TT(2), tud21 = TT(5), tuu12 = TT(6), tdu12 = TT(7), tuu22 = TT(8);
#undef TT
      da = cadd(da, cmul(tuu21, Cc));
      db = cadd(db, cmul(tud21, Cc));
      dc = cadd(dc, cadd(cadd(cmul(tuu12, A), cmul(tdu12, B)), cmul(tuu22, Cc)));
    }
    if (some) {
      const size_t i = P.nv + c;
      double2* LA = Lop + ((size_t)(a * 2 + 0) * nsl2 + la) * npad + i;
      double2* LB = Lop + ((size_t)(a * 2 + 1) * nsl2 + la) * npad + i;
      *LA = cadd(*LA, da);
      *LB = cadd(*LB, db);
    }
    C2lo[((size_t)a * nsl2 + la) * P.nlo + c] = dc;
  }
}

// ---------------------------------------------------------------------
// out(i,j) (+)= sum_k L[k][i] R[k][j] on the lower triangle i >= j, i, j < n
// (zher2m.f:69-80, 'L','N','T'): the FP64 HNS update, its LO-LO block and the
// adjoint's density matrices.  L, R k-major complex planes of row strides
// ldl, ldr (any); out column-major.
//
// Bound by the FP64 pipe (8 flops per element and k); the products run as
// m8n8k4 DMMA, which issues 256 FMA per instruction where a DFMA issues 32
// and so leaves the issue slots to the loads.  One block of 2 x 2 warps per
// 2 WT x 2 WT tile, WT x WT complex elements per warp (real and imaginary
// accumulators of (WT/8)^2 fragments, 4 DMMA per fragment and 4 k), the
// operand rows of TRI_KC k copied by cp.async three stages deep.  A row of
// shared memory holds 2 WT + 2 elements: the 8 lanes of a quarter-warp
// (4 k x 2 i) then read 8 different 16-byte banks.
// ---------------------------------------------------------------------
#define TRI_KC 16
#define TRI_STAGES 3
#define TRI_THREADS 128
__host__ __device__ constexpr int tri_smem_bytes(int wt) { return TRI_STAGES * 2 * TRI_KC * (2 * wt + 2) * 16; }

// 16-byte copy, or zeros when !in (src is not read then)
__device__ __forceinline__ void l1g_cp16z(void* dst, const void* src, bool in) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(in ? 16 : 0) : "memory");
}

// t0: the launch's first tile of the triangle in column order (columns of
// tiles left to right, each column's tiles bottom up); nb tiles per side.
// ovw: out is written instead of added to.  status: when non-null, a
// non-finite result sets L1G_STATUS_NONFINITE.
template <int WT>
__global__ void __launch_bounds__(TRI_THREADS, WT == 32 ? 2 : 4)
    k_tri_gemm(int n, int K, int nb, long t0, const double2* __restrict__ L, int ldl, const double2* __restrict__ R,
               int ldr, double2* __restrict__ out, int ld, int ovw, int* __restrict__ status) {
  constexpr int T = 2 * WT, F = WT / 8, RS = T + 2;  // tile side, fragments per warp side, smem row
  extern __shared__ double2 sm2[];
  // tile of this block: counted from the end, column c from the right holds c + 1 tiles
  const long tr = (long)nb * (nb + 1) / 2 - 1 - (t0 + blockIdx.x);
  long c = (long)((sqrt(8.0 * (double)tr + 1.0) - 1.0) * 0.5);
  while (c * (c + 1) / 2 > tr) c--;
  while ((c + 1) * (c + 2) / 2 <= tr) c++;
  const int j0 = (nb - 1 - (int)c) * T, i0 = (nb - 1 - (int)(tr - c * (c + 1) / 2)) * T;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wi = (warp & 1) * WT, wj = (warp >> 1) * WT;
  auto stage = [&](int k0) {
    double2* sL = sm2 + ((k0 / TRI_KC) % TRI_STAGES) * 2 * TRI_KC * RS;
    double2* sR = sL + TRI_KC * RS;
    for (int q = tid; q < TRI_KC * T; q += TRI_THREADS) {
      const int kk = q / T, r = q % T, k = k0 + kk;
      const bool il = k < K && i0 + r < n, ir = k < K && j0 + r < n;
      l1g_cp16z(sL + kk * RS + r, L + (il ? (size_t)k * ldl + i0 + r : 0), il);
      l1g_cp16z(sR + kk * RS + r, R + (ir ? (size_t)k * ldr + j0 + r : 0), ir);
    }
  };
  double re[F][F][2], im[F][F][2];
#pragma unroll
  for (int u = 0; u < F; u++)
#pragma unroll
    for (int v = 0; v < F; v++) re[u][v][0] = re[u][v][1] = im[u][v][0] = im[u][v][1] = 0.0;
  const int nk = (K + TRI_KC - 1) / TRI_KC;
#pragma unroll
  for (int q = 0; q < TRI_STAGES - 1; q++) {
    if (q < nk) stage(q * TRI_KC);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int q = 0; q < nk; q++) {
    asm volatile("cp.async.wait_group %0;" ::"n"(TRI_STAGES - 2) : "memory");
    __syncthreads();  // chunk q has landed; every warp is past chunk q - 1
    if (q + TRI_STAGES - 1 < nk) stage((q + TRI_STAGES - 1) * TRI_KC);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const double2* sL = sm2 + (q % TRI_STAGES) * 2 * TRI_KC * RS + (lane & 3) * RS + wi + (lane >> 2);
    const double2* sR = sm2 + (q % TRI_STAGES) * 2 * TRI_KC * RS + TRI_KC * RS + (lane & 3) * RS + wj + (lane >> 2);
#pragma unroll
    for (int k = 0; k < TRI_KC; k += 4) {
      double2 a[F], b[F];
#pragma unroll
      for (int u = 0; u < F; u++) a[u] = sL[k * RS + 8 * u];
#pragma unroll
      for (int v = 0; v < F; v++) b[v] = sR[k * RS + 8 * v];
#pragma unroll
      for (int u = 0; u < F; u++)
#pragma unroll
        for (int v = 0; v < F; v++) {
          dmma(re[u][v], a[u].x, b[v].x);
          dmma(im[u][v], a[u].x, b[v].y);
        }
#pragma unroll
      for (int u = 0; u < F; u++)
#pragma unroll
        for (int v = 0; v < F; v++) {
          dmma(re[u][v], -a[u].y, b[v].y);
          dmma(im[u][v], a[u].y, b[v].x);
        }
    }
  }
  // fragment element e of lane: row lane / 4, column 2 (lane % 4) + e
  bool bad = false;
#pragma unroll
  for (int v = 0; v < F; v++)
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const int j = j0 + wj + 8 * v + 2 * (lane & 3) + e;
      if (j >= n) continue;
      double2 o[F];
#pragma unroll
      for (int u = 0; u < F; u++) {
        const int i = i0 + wi + 8 * u + (lane >> 2);
        o[u] = (!ovw && i < n && i >= j) ? out[(size_t)j * ld + i] : cmk(0.0, 0.0);
      }
#pragma unroll
      for (int u = 0; u < F; u++) {
        const int i = i0 + wi + 8 * u + (lane >> 2);
        if (i >= n || i < j) continue;
        o[u] = cmk(o[u].x + re[u][v][e], o[u].y + im[u][v][e]);
        out[(size_t)j * ld + i] = o[u];
        bad |= l1g_nonfinite(o[u]);
      }
    }
  if (status && bad) atomicOr(status, L1G_STATUS_NONFINITE);
}

// LO block of HNS in split precision: HS(nv+i, nv+j) += T(i, j) on the lower
// triangle i >= j, T = C2^T CLM computed into a scratch block
__global__ void k_add_lower(int nv, int nlo, const double2* __restrict__ T, double2* __restrict__ hs, int ld,
                            int* __restrict__ status) {
  const int ci = blockIdx.x * blockDim.x + threadIdx.x;
  const int cj = blockIdx.y;
  if (ci >= nlo || ci < cj) return;
  double2* dst = hs + (size_t)(nv + cj) * ld + (nv + ci);
  const double2 v = cadd(*dst, T[(size_t)cj * nlo + ci]);
  *dst = v;
  if (status && l1g_nonfinite(v)) atomicOr(status, L1G_STATUS_NONFINITE);
}

// ---------------------------------------------------------------------
// K-orb: HORB (horb.F:98-297).  For U-atom a and l = lvor the reference adds
//   sum_(alpha,beta) g_(alpha beta) sum_(m0,m1) conj(X_alpha(m0,i)) pot(m1,m0) X_beta(m1,j)
// to HS(i,j), i >= j, with X = (ALM, BLM, CLM) of the row (CLM only on the
// atom type's own LO rows of that l, whose ALM, BLM are their LO coefficients;
// zero on all other LO rows) and g the overlaps of (u, udot, u_lo): g_AA =
// g_CC = 1, g_BB = PEI, g_AC = PI12LO, g_BC = PE12LO.  (Its cases PW-PW, PW-LO
// and LO-LO are this sum with the zero parts left out: i >= j puts an LO row j
// of the same type and l in a block not after i's.)  So all atoms and l
// together are one product over k = (item, alpha, m0), L[k][i] = conj(X), R[k][j]
// = the inner sums, which k_tri_gemm adds in one pass over HS.
// ---------------------------------------------------------------------
struct OrbItem {
  int a, lvor, pot, k0;  // atom, l, its pot(m2,m1) block of 49, first k
};
__global__ void k_horb_rows(DevProb P, const OrbItem* __restrict__ items, const double2* __restrict__ pots,
                            const LoRange* __restrict__ lor, int nlor, double2* __restrict__ L,
                            double2* __restrict__ R) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= P.n) return;
  const OrbItem it = items[blockIdx.y];
  const int a = it.a, lvor = it.lvor, nm = 2 * lvor + 1;
  const double2* pot = pots + (size_t)it.pot * 49;  // [7][7] pot(m2,m1)
  const int jn = P.atype[a];
  const double pi = 3.141592653589793238462643;
  const double rhoatm = 4.0 * pi * sqrt(P.vi) * P.rmt[jn] * P.rmt[jn];
  const double* r = P.pos + 3 * a;
  const double2 ph = cexp2pi(r[0] * P.kzz[3 * i] + r[1] * P.kzz[3 * i + 1] + r[2] * P.kzz[3 * i + 2]);
  double2 y[16];
  dev_ylm_row<3>(P.xk[i], P.yk[i], P.zk[i], P.rotij + 9 * a, P.rotloc + 9 * jn, lvor, y);
  double2 cil = cmk(1.0, 0.0);
  for (int q = 0; q < lvor; q++) cil = cmk(-cil.y, cil.x);
  // the row's coefficients of (u, udot, u_lo): X = coefficient times t(m)
  double ca = 0.0, cb = 0.0, cc = 0.0;
  if (i < P.nv) {
    const size_t o = ((size_t)jn * P.ltop + lvor) * P.nvpad + i;
    ca = P.al[o];
    cb = P.bl[o];
  } else {
    const int li = i - P.nv + 1;
    int myjlo = 0;
    for (int q = 0; q < nlor; q++)
      if (lor[q].jn == jn && lor[q].l == lvor && li >= lor[q].i1 && li <= lor[q].i2) myjlo = lor[q].jlo;
    if (myjlo > 0) {
      const int oo = (jn * L1G_NLOAT + myjlo - 1) * (L1G_LOMAX + 1) + lvor;
      ca = P.alo[oo];
      cb = P.blo[oo];
      cc = P.clo[oo];
    }
  }
  const double peil = P.pei[jn * P.ldl + lvor];
  const double pi12 = lvor <= L1G_LOMAX ? P.pi12lo[jn * (L1G_LOMAX + 1) + lvor] : 0.0;
  const double pe12 = lvor <= L1G_LOMAX ? P.pe12lo[jn * (L1G_LOMAX + 1) + lvor] : 0.0;
  const double ga = ca + pi12 * cc, gb = peil * cb + pe12 * cc, gc = pi12 * ca + pe12 * cb + cc;
  const size_t st = P.npad;
  double2* Li = L + (size_t)it.k0 * st + i;
  double2* Ri = R + (size_t)it.k0 * st + i;
  double2 t[7];
#pragma unroll
  for (int m = 0; m < 7; m++)
    if (m < nm) t[m] = cmul(cmul(cscale(cil, rhoatm), ph), cconj(y[lvor * lvor + m]));
#pragma unroll
  for (int m0 = 0; m0 < 7; m0++) {
    if (m0 >= nm) continue;
    double2 q = cmk(0.0, 0.0);  // sum_m1 pot(m1,m0) t(m1)
#pragma unroll
    for (int m1 = 0; m1 < 7; m1++)
      if (m1 < nm) q = cadd(q, cmul(pot[(m1 + 3 - lvor) * 7 + m0 + 3 - lvor], t[m1]));
    const double2 tc = cconj(t[m0]);
    Li[(size_t)m0 * st] = cscale(tc, ca);
    Li[(size_t)(nm + m0) * st] = cscale(tc, cb);
    Li[(size_t)(2 * nm + m0) * st] = cscale(tc, cc);
    Ri[(size_t)m0 * st] = cscale(q, ga);
    Ri[(size_t)(nm + m0) * st] = cscale(q, gb);
    Ri[(size_t)(2 * nm + m0) * st] = cscale(q, gc);
  }
}

// non-finite scan of the n x n block and hsdiag (hsdiag may be null)
__global__ void k_check_finite(int n, const double2* __restrict__ hs, int ld, const double2* __restrict__ hsdiag,
                               int* status) {
  // a component is non-finite when its exponent bits are all ones
  unsigned bad = 0;
  for (int j = blockIdx.x; j < n; j += gridDim.x) {
    const double2* col = hs + (size_t)j * ld;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const double2 v = col[i];
      bad |= ((unsigned)(__double_as_longlong(v.x) >> 52) & 0x7ffu) == 0x7ffu;
      bad |= ((unsigned)(__double_as_longlong(v.y) >> 52) & 0x7ffu) == 0x7ffu;
    }
  }
  if (blockIdx.x == 0 && hsdiag)
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const double2 d = hsdiag[i];
      bad |= ((unsigned)(__double_as_longlong(d.x) >> 52) & 0x7ffu) == 0x7ffu;
      bad |= ((unsigned)(__double_as_longlong(d.y) >> 52) & 0x7ffu) == 0x7ffu;
    }
  if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(status, L1G_STATUS_NONFINITE);
}

// The generalized problem SECLR4 solves (seclr4.F:158-345), unpacked from
// the packed state: H(i,j) = conj(HS(i,j)) and S(i,j) = conj(HS(j,i)) for
// i > j (ZHCGST factors S**T), real diagonals from HS(i,i) and HSDIAG(i);
// the lower triangles of H and S, column-major n x n (ld n).
__global__ void k_unpack_seclr(int n, const double2* __restrict__ hs, int ld, const double2* __restrict__ hsdiag,
                               double2* __restrict__ H, double2* __restrict__ S) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;  // row
  const int j = blockIdx.y;                             // column
  if (i >= n || i < j) return;
  const size_t o = (size_t)j * n + i;
  if (i == j) {
    H[o] = cmk(hs[(size_t)i * ld + i].x, 0.0);
    S[o] = cmk(hsdiag[i].x, 0.0);
  } else {
    H[o] = cconj(hs[(size_t)j * ld + i]);
    S[o] = cconj(hs[(size_t)i * ld + j]);
  }
}
