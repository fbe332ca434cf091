// fsp_tc.cuh -- the adjoint's spherical pairs of two different row blocks as
// int8 projections on the tensor cores (split precision), sm_100a.
//
// forces.cuh derives the projections: per atom a of type t and per (alpha, lm),
//   P_alpha = sum_J A^alpha_(t l)(J) Z_lm(J) y_b(J),  y_b(J) = conj(phi_a(J)) c_b(J),
// and the same with the weights kappa_g(J) = 2 pi KZZ_g(J), g = 1..3.  A Z kappa
// is real, so per atom this is a real-by-complex product
//   rows (lm, alpha, g)   : A^alpha Z_lm {1, kappa_1, kappa_2, kappa_3}  (of the type)
//   columns (b, re | im)  : Re, Im y_b                                    (of the atom)
// with half the multiplications of the complex product of A Z conj(phi_a) with
// (G c), whose left operand is complex.  Both operands are cut into S int8
// slices per row block (power-of-two scales per row and block).
//
// One CTA forms a tile of 16 lm (128 rows: 8 consecutive rows per lm, alpha 4 +
// g) x NB bands for all row blocks in turn.  After block p its epilogue
// contracts the block's projections Y with the running sum of the blocks
// before, the prefix, which stays in registers, and adds Y to it: the 2x2 forms
// over (alpha, beta) and the products of g = 0 with g = 1..3 combine the 8 rows
// of an lm, which are 8 lanes of one warp.  Nothing but three sums per CTA goes
// back to memory.
//
// Bound by the tensor core: S (S+1)/2 products of K = block rows, 128 x N per
// block.  Only the epilogue's TMEM reads stall the MMAs (the next block needs
// the same accumulators); the contraction runs beside the next block's.
// Measured at 100 atoms, NV = 11777, 400 bands, 6 slices, blocks of 1024 rows:
// products 15.4 ms (2.9e15 int8 ops/s with the padding; tensor pipe active 64%
// of the time), operands 3.7 and 2.5, in three pieces of atoms;
// the complex products over blocks, their slicing, k-major left operand and
// prefix kernel before took 38.  The operands are bound by the integer work of
// cutting 1.7e9 values into 6 digits (2.1 TB/s of stores).
#pragma once

namespace fsptc {

using split::desc_sw64;
using split::digit7;
using split::elect_one;
using split::idesc_i8;
using split::mbar_expect_tx;
using split::mbar_init;
using split::mbar_try_wait;
using split::mbar_wait;
using split::mma_commit;
using split::mma_i8;
using split::pow2_exact;
using split::smem_u32;
using split::tc_fence_after;
using split::tc_fence_before;
using split::tma_load_3d;
using sphtc::Ring;
using sphtc::wait_or_abort;

constexpr int LMT = 16;  // lm per tile (128 rows)

template <int S>
struct Cfg {
  // real columns: at most 80 (prefix and block values of 40 columns per
  // epilogue thread), S levels of them in 512 TMEM columns
  static constexpr int NFIT = ((512 / S) / 16) * 16;
  static constexpr int N = NFIT > 80 ? 80 : NFIT;
  static constexpr int NB = N / 2;   // bands per tile
  static constexpr int HB = NB / 2;  // bands per epilogue thread (column halves)
  static_assert(HB % 2 == 0, "two bands per TMEM load");
  static constexpr int A_BYTES = S * 128 * 64, B_BYTES = S * N * 64, STAGE = A_BYTES + B_BYTES;
  static constexpr int FIT = (220 * 1024) / STAGE;
  static constexpr int STAGES = FIT > 4 ? 4 : FIT;
  static_assert(STAGES >= 2, "the ring needs two stages");
  static constexpr int SMEM = STAGES * STAGE + 1024;
  // 8 epilogue warps, then the MMA warp, the TMA warp and two idle ones (the
  // register split is per warpgroup): 384 threads launch with 168 registers,
  // 224 x 256 + 56 x 128 is the same total
  static constexpr int EPI = 256, THREADS = EPI + 128, REPI = 224, RMISC = 56;
  static_assert(REPI * EPI + RMISC * 128 <= 168 * THREADS, "register split above the launch's registers");
};

// Z_lm of every PW row: zt[lm][J] (row stride nvpad)
__global__ void k_fsp_zlm(DevProb P, double* __restrict__ zt) {
  const int J = blockIdx.x * blockDim.x + threadIdx.x, lm = blockIdx.y;
  if (J >= P.nv) return;
  double ux = 0.0, uy = 0.0, uz = 1.0;
  const double r = P.rk[J];
  if (r > 0.0) {
    ux = P.xk[J] / r;
    uy = P.yk[J] / r;
    uz = P.zk[J] / r;
  }
  const int l = frc_lof(lm);
  zt[(size_t)lm * P.nvpad + J] = frc_zlm(ux, uy, uz, l, lm - l * l - l);
}

// sum_d c_d 2^(-7d) over the S levels of one accumulator element: three
// levels at a time combined exactly in int64 (|c| < 2^31, so a triple lies
// below 2^46) and converted by one add (1.5 2^52 + V has V in its low mantissa
// bits for |V| < 2^51), then the triples in FP64: 3 FP64 operations at 6 slices
// where level by level they are 12
template <int S>
__device__ __forceinline__ double level_sum3(const uint32_t (&r)[S]) {
  constexpr int last = (S - 1) / 3 * 3;
  double v = 0.0;
#pragma unroll
  for (int d0 = last; d0 >= 0; d0 -= 3) {  // the smallest levels first
    const int cnt = S - d0 < 3 ? S - d0 : 3;
    long long t = (long long)(int)r[d0];
#pragma unroll
    for (int d = 1; d < cnt; d++) t = t * 128 + (long long)(int)r[d0 + d];
    const double x = __longlong_as_double(t + 0x4338000000000000LL) - 6755399441055744.0;
    const double w = 1.0 / (double)(1LL << (7 * (d0 + cnt - 1)));
    v = d0 == last ? x * w : fma(x, w, v);
  }
  return v;
}

// The power of two 2^(6 - e + 7 (S-1)) that turns a row of exponent e into
// integers of S digits, as two exact factors (each in range for every e)
struct DigitScale {
  double a, b;
};
template <int S>
__device__ __forceinline__ DigitScale digits_scale(int e) {
  const int k = 6 - e + 7 * (S - 1), h = k / 2;
  return {pow2_exact(h), pow2_exact(k - h)};
}
// Four consecutive values of one row cut into S int8 digits, one 32-bit store
// per slice.  Each value is rounded to an integer V, |V| <= 2^(7 S - 1), by one
// FMA onto 1.5 2^52; with 64 added to every digit below the first, the digits
// of V are 7-bit fields (0..127, the offset taken off again four bytes at a
// time): integer work where the digit-by-digit cut costs four FP64 operations
// each (24 per value, which took 5.0 and 2.8 ms for the two operands at 100
// atoms).  8 slices (V beyond 2^51) keep that cut.
template <int S>
__device__ __forceinline__ void store_digits(const double (&v)[4], const DigitScale& sc, int8_t* out, size_t plane) {
  if (S <= 7) {
    long long off = 0;
    for (int p = 0; p + 1 < S; p++) off = off * 128 + 64;
    long long V[4];
#pragma unroll
    for (int q = 0; q < 4; q++)
      V[q] = __double_as_longlong(fma(v[q] * sc.a, sc.b, 6755399441055744.0)) - 0x4338000000000000LL + off;
#pragma unroll
    for (int p = 0; p < S; p++) {
      const int sh = 7 * (S - 1 - p);
      uint32_t w = 0;
#pragma unroll
      for (int q = 0; q < 4; q++) w |= ((uint32_t)(V[q] >> sh) & (p ? 0x7fu : 0xffu)) << (8 * q);
      if (p) w = ((w | 0x80808080u) - 0x40404040u) ^ 0x80808080u;  // per byte: minus 64
      *reinterpret_cast<uint32_t*>(out + (size_t)p * plane) = w;
    }
  } else {
    double t[4];
#pragma unroll
    for (int q = 0; q < 4; q++) t[q] = v[q] * sc.a * sc.b * (1.0 / (double)(1LL << (7 * (S - 1))));
#pragma unroll
    for (int p = 0; p < S; p++) {
      uint32_t w = 0;
#pragma unroll
      for (int q = 0; q < 4; q++) w |= (uint32_t)(digit7(t[q]) & 0xff) << (8 * q);
      *reinterpret_cast<uint32_t*>(out + (size_t)p * plane) = w;
    }
  }
}

// Left operand of one (row block, lm, type): rows (type, lm, alpha 4 + g),
// out [S][rows][Kp], the block's rows at columns blk fBp ..; ex [rows][nblk].
// lm past ltop^2 (the last tile's rest) are zero rows.
template <int S>
__global__ void __launch_bounds__(256, 2) k_fsp_left(DevProb P, const double* __restrict__ zt, int t0, int fB, int fBp,
                                                  int Kp, size_t rows, int8_t* __restrict__ out,
                                                  int* __restrict__ ex, int* __restrict__ status) {
  __shared__ double red[8][8];
  __shared__ int se[8];
  const int blk = blockIdx.x, lm = blockIdx.y, t = t0 + blockIdx.z, nblk = gridDim.x;
  const int J0 = blk * fB, kc = min(fB, P.nv - J0);
  const bool pad = lm >= P.ltop * P.ltop;
  const int l = pad ? 0 : frc_lof(lm);
  const double* al = P.al + ((size_t)t * P.ltop + l) * P.nvpad + J0;
  const double* bl = P.bl + ((size_t)t * P.ltop + l) * P.nvpad + J0;
  const double* z = zt + (size_t)(pad ? 0 : lm) * P.nvpad + J0;
  const int* kz = P.kzz + 3 * (size_t)J0;
  auto row = [&](int j, double(&a)[2], double(&kap)[4]) {  // {AL, BL} Z and {1, kappa} of block row j
    const bool in = j < kc && !pad;
    const double zz = in ? z[j] : 0.0;
    a[0] = in ? al[j] * zz : 0.0;
    a[1] = in ? bl[j] * zz : 0.0;
    kap[0] = 1.0;
#pragma unroll
    for (int c = 0; c < 3; c++) kap[c + 1] = in ? FRC_2PI * kz[3 * j + c] : 0.0;
  };
  double m[8] = {};
  bool bad = false;
  for (int j = threadIdx.x; j < kc; j += 256) {
    double a[2], kap[4];
    row(j, a, kap);
#pragma unroll
    for (int r = 0; r < 8; r++) m[r] = fmax(m[r], fabs(a[r >> 2] * kap[r & 3]));
    bad |= l1g_nonfinite(make_double2(a[0], a[1]));
  }
  if (bad) atomicOr(status, L1G_STATUS_NONFINITE);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int r = 0; r < 8; r++) {
    double v = m[r];
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (lane == 0) red[warp][r] = v;
  }
  __syncthreads();
  const size_t row0 = ((size_t)blockIdx.z * gridDim.y + lm) * 8;
  if (threadIdx.x < 8) {
    double v = 0.0;
    for (int w = 0; w < 8; w++) v = fmax(v, red[w][threadIdx.x]);
    const int e = v > 0.0 ? ilogb(v) + 1 : 0;
    se[threadIdx.x] = e;
    ex[(row0 + threadIdx.x) * nblk + blk] = e;
  }
  __syncthreads();
  const size_t plane = rows * Kp;
  for (int j = 4 * threadIdx.x; j < fBp; j += 4 * 256) {
    double a0[4], a1[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      double a[2], kap[4];
      row(j + q, a, kap);
      a0[q] = a[0];
      a1[q] = a[1];
    }
#pragma unroll 1
    for (int r = 0; r < 8; r++) {  // a row's digits at a time (all 8 together take 250 registers)
      const int g = r & 3;
      double v[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const double x = r < 4 ? a0[q] : a1[q];
        v[q] = (g && j + q < kc) ? x * (FRC_2PI * kz[3 * (j + q) + g - 1]) : x;
      }
      store_digits<S>(v, digits_scale<S>(se[r]), out + (row0 + r) * Kp + (size_t)blk * fBp + j, plane);
    }
  }
}

// exponents of the right operand, ex[band][block]: |Re y|, |Im y| <= |c|, the
// same for every atom
__global__ void __launch_bounds__(256) k_fsp_cexp(int nv, int nb, int fB, const double2* __restrict__ C, int ldc,
                                                  int* __restrict__ ex) {
  __shared__ double red[8];
  const int blk = blockIdx.x, b = blockIdx.y, J0 = blk * fB, kc = min(fB, nv - J0);
  double m = 0.0;
  for (int j = threadIdx.x; j < kc; j += 256) {
    const double2 c = C[(size_t)b * ldc + J0 + j];
    m = fmax(m, hypot(c.x, c.y));
  }
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; w++) m = fmax(m, red[w]);
    ex[(size_t)b * gridDim.x + blk] = m > 0.0 ? ilogb(m) + 1 : 0;
  }
}

// Right operand of one (row block, 8 bands, atom): rows (atom, band, re | im),
// bands past nb zero; layout as the left one's
template <int S>
__global__ void __launch_bounds__(256, 2) k_fsp_right(DevProb P, const double2* __restrict__ C, int ldc, int nb, int nbp,
                                                   int a0, int fB, int fBp, int Kp, size_t rows,
                                                   const int* __restrict__ exC, int8_t* __restrict__ out,
                                                   int* __restrict__ status) {
  const int blk = blockIdx.x, a = a0 + blockIdx.z, nblk = gridDim.x;
  const int J0 = blk * fB, kc = min(fB, P.nv - J0);
  const size_t plane = rows * Kp;
  bool bad = false;
  for (int j = 4 * threadIdx.x; j < fBp; j += 4 * 256) {
    double2 ph[4];
#pragma unroll
    for (int q = 0; q < 4; q++) ph[q] = j + q < kc ? P.phase[(size_t)a * P.npad + J0 + j + q] : cmk(0.0, 0.0);
    for (int b = blockIdx.y * 8; b < min(nbp, (int)blockIdx.y * 8 + 8); b++) {
      double re[4], im[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const double2 c = (b < nb && j + q < kc) ? C[(size_t)b * ldc + J0 + j + q] : cmk(0.0, 0.0);
        const double2 y = cmul(cconj(ph[q]), c);
        re[q] = y.x;
        im[q] = y.y;
        bad |= l1g_nonfinite(y);
      }
      const DigitScale sc = digits_scale<S>(b < nb ? exC[(size_t)b * nblk + blk] : 0);
      int8_t* o = out + ((size_t)blockIdx.z * 2 * nbp + 2 * b) * Kp + (size_t)blk * fBp + j;
      store_digits<S>(re, sc, o, plane);
      store_digits<S>(im, sc, o + Kp, plane);
    }
  }
  if (bad) atomicOr(status, L1G_STATUS_NONFINITE);
}

// Products and contraction.  CTA: band tile x, lm tile y, atom a0 + z; the left
// operand's rows start at type t0.
template <int S>
__global__ void __launch_bounds__(Cfg<S>::THREADS, 1)
    k_fsp_gemm(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, DevProb P,
               const SphCoef* __restrict__ coef, int a0, int t0, int nblk, int fB, int fBp, int nb, int nbp,
               const int* __restrict__ exA, const int* __restrict__ exC, const double* __restrict__ f,
               const double* __restrict__ eps, double* __restrict__ F, int* __restrict__ status, int never_wait) {
  using C = Cfg<S>;
  constexpr int N = C::N, STAGES = C::STAGES, HB = C::HB;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full[STAGES], empty[STAGES], tfull, tempty, accbar, never;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  __shared__ double sf[C::NB], sfe[C::NB], red[8][3];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // warp-uniform to the compiler
  const int bt = blockIdx.x, mt = blockIdx.y, az = blockIdx.z, a = a0 + az, t = P.atype[a];
  const int ra0 = ((t - t0) * (int)gridDim.y + mt) * 128, rb0 = az * 2 * nbp + bt * N;
  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int s = 0; s < STAGES; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(&tfull, 1);
    mbar_init(&tempty, 8);  // one arrival per epilogue warp
    mbar_init(&accbar, 1);
    mbar_init(&never, 1);  // nothing arrives here (the never_wait test hook)
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  for (int q = tid; q < C::NB; q += C::THREADS) {
    const int b = bt * C::NB + q;
    sf[q] = b < nb ? f[b] : 0.0;
    sfe[q] = b < nb ? f[b] * eps[b] : 0.0;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  // 64-row K blocks of row block p
  auto kblocks = [&](int p) { return (min(fB, P.nv - p * fB) + 63) / 64; };

  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::RMISC));
    if (warp == 9) {
      // ---- TMA producer, a full ring ahead of the MMAs ----
      if (lane == 0) {
        Ring<STAGES> r;
        int n = 0;  // stages issued, up to a full ring
        bool ok = true;
        for (int p = 0; p < nblk && ok; p++) {
          const int nkb = kblocks(p);
          for (int kb = 0; kb < nkb; kb++) {
            if (n == STAGES && !wait_or_abort(&empty[r.slot], r.par ^ 1, &abort_flag)) {
              ok = false;
              break;
            }
            uint8_t* s = smem + r.slot * C::STAGE;
            mbar_expect_tx(&full[r.slot], C::STAGE);
            tma_load_3d(s, &tmA, &full[r.slot], p * fBp + kb * 64, ra0, 0);
            tma_load_3d(s + C::A_BYTES, &tmB, &full[r.slot], p * fBp + kb * 64, rb0, 0);
            r.next();
            if (n < STAGES) n++;
          }
        }
        if (!ok) atomicOr(status, L1G_STATUS_TIMEOUT);
        // the copies in flight land before the shared memory is released
        for (int q = 0; q < n; q++) {
          const int st = (r.slot + STAGES - 1 - q) % STAGES;
          mbar_wait(&full[st], st < r.slot ? r.par : r.par ^ 1);
        }
      }
      __syncwarp();
    } else if (warp == 8) {
      // ---- MMA issuer: a converged warp, one elected lane issues ----
      Ring<STAGES> r;
      bool ok = true;
      auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
        return __all_sync(0xffffffffu, wait_or_abort(bar, parity, &abort_flag));
      };
      if (never_wait) ok = __all_sync(0xffffffffu, sphtc::never_arrives(&never));
      const uint64_t desc0 = desc_sw64(smem_u32(smem));
      for (int p = 0; p < nblk && ok; p++) {
        if (p > 0) ok = wait(&tempty, (uint32_t)(p - 1) & 1);
        const int nkb = kblocks(p);
        for (int kb = 0; kb < nkb && ok; kb++) {
          ok = wait(&full[r.slot], r.par);
          if (!ok) break;
          tc_fence_after();
          const uint64_t ad0 = desc0 + (uint32_t)(r.slot * (C::STAGE >> 4)), bd0 = ad0 + (C::A_BYTES >> 4);
          if (elect_one()) {
            // as k_split_gemm: A slice p times B slices q0.. is one MMA of at
            // most 256 columns, landing on consecutive levels
            constexpr int QC = (256 / N) < S ? (256 / N) : S;
#pragma unroll
            for (int sa = 0; sa < S; sa++)
#pragma unroll
              for (int q0 = 0; q0 < S - sa; q0 += QC)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                  const int cnt = (S - sa - q0) < QC ? (S - sa - q0) : QC;
                  mma_i8(tmem + (uint32_t)((sa + q0) * N), ad0 + ((sa * 128 * 64 + h * 32) >> 4),
                         bd0 + ((q0 * N * 64 + h * 32) >> 4), idesc_i8(128, cnt * N),
                         (h > 0 || sa > 0) ? 1u : (uint32_t)(kb > 0));
                }
            mma_commit(&empty[r.slot]);
            if (kb == nkb - 1) mma_commit(&tfull);
          }
          __syncwarp();
          r.next();
        }
      }
      if (elect_one()) {
        if (!ok) {
          atomicOr(status, L1G_STATUS_TIMEOUT);
          *(volatile int*)&abort_flag = 1;
        }
        mma_commit(&accbar);
      }
    }
    __syncwarp();
  } else {
    // ---- epilogue warps: row 32 (w % 4) + lane, column half w / 4 ----
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(C::REPI));
    const int row = 32 * (warp & 3) + lane, hb = (warp >> 2) * HB;
    const int lm = mt * LMT + (row >> 3), al = (lane >> 2) & 1;
    const uint32_t trow = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(2 * hb);
    // this row's part of the 2x2 forms: MY_alpha = wd Y_alpha + wo Y_(other alpha)
    double hd = 0.0, ho = 0.0, sd = 0.0;
    if (lm < P.ltop * P.ltop) {
      const SphCoef cf = coef[t * P.ltop + frc_lof(lm)];
      hd = cf.vif * (al ? cf.mBB : cf.mAA);
      ho = cf.vif * (al ? cf.mBA : cf.mAB);
      sd = al ? cf.vif * cf.chn : cf.vif;
    }
    double2 Pre[HB], Y[HB];
#pragma unroll
    for (int q = 0; q < HB; q++) Pre[q] = cmk(0.0, 0.0);
    double acc = 0.0;
    bool ok = true;
    for (int p = 0; p < nblk; p++) {
      const double sa = pow2_exact(exA[(size_t)(ra0 + row) * nblk + p] - 12);
      if (!__all_sync(0xffffffffu, wait_or_abort(&tfull, (uint32_t)p & 1, &abort_flag)) ||
          __any_sync(0xffffffffu, *(volatile int*)&abort_flag)) {
        ok = false;
        break;
      }
      tc_fence_after();
#pragma unroll
      for (int q = 0; q < HB; q += 2) {
        uint32_t r[S][4];
        sphtc::tmem_ld4<S>(r, trow + 2 * q, N);
        const int b = bt * C::NB + hb + q;
        const double s0 = sa * pow2_exact(b < nb ? exC[(size_t)b * nblk + p] : 0),
                     s1 = sa * pow2_exact(b + 1 < nb ? exC[(size_t)(b + 1) * nblk + p] : 0);
        sphtc::tmem_wait4<S>(r);
        double v[4];
#pragma unroll
        for (int m = 0; m < 4; m++) {
          uint32_t rr[S];
#pragma unroll
          for (int d = 0; d < S; d++) rr[d] = r[d][m];
          v[m] = level_sum3<S>(rr);
        }
        Y[q] = cmk(v[0] * s0, v[1] * s0);
        Y[q + 1] = cmk(v[2] * s1, v[3] * s1);
      }
      // every column read: the next block's MMAs may start
      tc_fence_before();
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&tempty)) : "memory");
      if (p > 0) {
        const int l0 = lane & ~3;  // the lane of g = 0 with this lm and alpha
#pragma unroll
        for (int q = 0; q < HB; q++) {
          const double fb = sf[hb + q], wd = fma(fb, hd, -(sfe[hb + q] * sd)), wo = fb * ho;
          const double2 yo = cmk(__shfl_xor_sync(0xffffffffu, Y[q].x, 4), __shfl_xor_sync(0xffffffffu, Y[q].y, 4));
          const double2 my = cmk(fma(wd, Y[q].x, wo * yo.x), fma(wd, Y[q].y, wo * yo.y));
          const double2 p0 = cmk(__shfl_sync(0xffffffffu, Pre[q].x, l0), __shfl_sync(0xffffffffu, Pre[q].y, l0));
          const double2 m0 = cmk(__shfl_sync(0xffffffffu, my.x, l0), __shfl_sync(0xffffffffu, my.y, l0));
          // Im(P_0 conj(MY_g)) - Im(P_g conj(MY_0)); zero for g = 0
          acc += fma(p0.y, my.x, -(p0.x * my.y)) - fma(Pre[q].y, m0.x, -(Pre[q].x * m0.y));
        }
      }
#pragma unroll
      for (int q = 0; q < HB; q++) Pre[q] = cadd(Pre[q], Y[q]);
    }
    if (!ok) {
      *(volatile int*)&abort_flag = 1;
      if (lane == 0) atomicOr(status, L1G_STATUS_TIMEOUT);
    }
    // sums over alpha and the warp's lm: lanes 1..3 hold the components
    acc += __shfl_xor_sync(0xffffffffu, acc, 4);
    acc += __shfl_xor_sync(0xffffffffu, acc, 8);
    acc += __shfl_xor_sync(0xffffffffu, acc, 16);
    if (lane >= 1 && lane < 4) red[warp][lane - 1] = acc;
  }
  if (warp == 8) mbar_wait(&accbar, 0);  // every MMA issued has completed before TMEM is freed
  tc_fence_before();
  __syncthreads();
  if (tid < 3) {
    double v = 0.0;
    for (int w = 0; w < 8; w++) v += red[w][tid];
    atomicAdd(&F[a * 3 + tid], -2.0 * v);
  }
  if (warp == 8) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

}  // namespace fsptc
