// sph_tc.cuh -- the spherical muffin-tin part of H and S (hamilt.F:371-440)
// on the 5th-generation tensor cores, split precision, sm_100a.
//
// For a pair (J <= I) HAMILT accumulates, per atom type and l,
//   S(J,I) += PHASE(J,I) (2l+1) P_l(x_JI) VIF [AL_J AL_I + CHN BL_J BL_I]
// and the same with the non-symmetric 2x2 block for H.  With PHASE =
// sum_eq phi_a(J) conj(phi_a(I)) the type and equivalent-atom sums at fixed
// l are one complex GEMM over k = (atom a, r in {AL, BL}):
//   G_l(J, I) = sum_k u_l(J,k) conj(v_l(I,k)),
//   u_l(J, (a,r)) = phi_a(J) {AL, BL}_(type a, l, J),
//   v_l(I, (a,r)) = phi_a(I) VIF {AL, CHN BL} (S) or VIF {hA, hB} (H),
// and the Legendre weight w_l(J,I) = (2l+1) P_l(x_JI), which couples J and I
// non-separably, is applied per pair as G_l leaves the accumulator:
//   aS(J,I) = sum_l w_l(J,I) G^S_l(J,I), aH likewise.
// The GEMMs run as Ozaki int8 slice products (the scheme of split_tc.cuh:
// power-of-two row scales, S slices, one exact int32 TMEM accumulator per
// level p+q-2 < S) with kind::i8 tcgen05.mma, M = 128 rows J, N = 4 real
// columns per I (S re, S im, H re, H im).  The accumulator is double
// buffered over l (2 x S levels x N columns of TMEM), so the FP64 epilogue
// of l (combine levels, scale, weight, accumulate per pair in registers)
// overlaps the MMAs of l+1.  After the last l the interstitial terms are
// gathered from the Theta/WARP table and HS is written as k_spherical does.
//
// Warp roles: warps 0..4 EG-1 epilogue (warp w reads TMEM lanes 32 (w%4)..
// and the I group w/4 of 4 I), warp 4 EG issues the MMAs, warp 4 EG + 1 lane 0
// the TMA loads (a full ring ahead of the MMAs, whatever they wait on).  Every
// mbarrier wait is bounded; a timeout sets a status bit and ends the CTA's
// work cleanly (copies drained, MMAs complete, TMEM freed).
//
// What bounds it, by the MMA issuer's clocks (5 slices, 64-byte K blocks): at
// 100 atoms (13 K steps per l) 66% in issuing, behind the tensor core's queue,
// 29% in waits for operands, 5% for a free accumulator; at 40 atoms (5 K steps)
// 53, 21 and 26%.  The tensor pipe is active 53 and 39% of the time.  Issued by one lane in a branch of its own, an MMA
// took 110 clocks of that lane against 77 on the tensor core, and the scales
// of the epilogue (Legendre weight, exponents) 580 clocks per pair and l
// behind the TMEM loads; with the issue from a converged warp, the scales
// formed before the wait for the accumulator, explicit polynomials and the
// tile's rows in shared memory, 40 atoms (N = 4937) went from 1.69 to 1.33 ms
// and 100 atoms (N = 12677) from 38.0 to 30.2 Mclk, 22.0 to 20.4-21.6 ms: the
// power cap sets the clock there.  A tile of two 12-I halves that share each A
// block (36% less feed, 8 pairs per epilogue thread by a register split) took
// the same time and was not kept (which of the shares grew instead was not
// recorded), nor did row pitches of 64 or 128 bytes help.
#pragma once
#include "legendre.cuh"

namespace sphtc {

using split::desc_kblock;
using split::digit7;
using split::digit_scale;
using split::elect_one;
using split::i2d_exact;
using split::idesc_i8;
using split::mbar_expect_tx;
using split::mbar_init;
using split::mbar_try_wait;
using split::mbar_wait;
using split::mma_commit;
using split::mma_i8;
using split::smem_u32;
using split::tc_fence_after;
using split::tc_fence_before;
using split::tma_load_3d;

// KB: bytes of K per pipeline stage and row (64: 64-byte swizzled rows, a
// deep ring; 128: 128-byte swizzled rows, half the TMA row requests per
// byte, two stages) -- a tunable tile shape
template <int S, int KB = 64>
struct Cfg {
  // real columns per level of one accumulator buffer: 4 per I, at most 48
  // (12 I: three epilogue warp groups of 4 I)
  static constexpr int NMAX = ((512 / (2 * S)) / 16) * 16;
  static constexpr int N = NMAX > 48 ? 48 : NMAX;
  static_assert(S * N <= 256, "one MMA per A slice needs (S - p) N <= 256 columns");
  static constexpr int IT = N / 4;   // I per tile
  static constexpr int IPT = 4;      // I per epilogue thread
  static constexpr int EG = IT / IPT;  // epilogue warp groups (4 warps each: the 4 TMEM lane quarters)
  static_assert(EG * IPT == IT, "I per tile must be a multiple of 4");
  static constexpr int EPI = 128 * EG;  // epilogue threads
  // one pipeline stage: all S slices of a KB-byte K block of A (128 rows)
  // and of B (N rows)
  static_assert(KB == 64 || KB == 128, "K block of 64 or 128 bytes");
  static constexpr int KSTEPS = KB / 32;  // 32-byte MMA K steps per stage
  static constexpr int A_BYTES = S * 128 * KB;
  static constexpr int B_BYTES = S * N * KB;
  // per-tile tables: exponents eA - 12 per (l, J) and eB per (l, I, S|H) as
  // int16, and the rows of the tile's I (unit vector, length, KZZ)
  static constexpr int SCALE_BYTES = (SPH_LMAX * 128 + SPH_LMAX * 2 * IT) * 2;
  static constexpr int ROW_BYTES = IT * 48;
  static constexpr int ROOM = 227 * 1024 - SCALE_BYTES - ROW_BYTES - 1024;
  static constexpr int STAGE = A_BYTES + B_BYTES;
  static constexpr int STAGES_FIT = ROOM / STAGE;
  static constexpr int STAGES = STAGES_FIT > 8 ? 8 : STAGES_FIT;
  static_assert(STAGES >= 2, "the ring needs two stages");
  static constexpr int SMEM = STAGES * STAGE + SCALE_BYTES + ROW_BYTES + 1024;
  static constexpr int THREADS = EPI + 64;  // + the MMA warp and the TMA warp
};

// Operand rows of one l, built from AL/BL, phases and the per-(type, l)
// coefficients, then cut into S int8 slices with a power-of-two scale per
// complex row.  isB = 0: complex row J -> real row J = [Re u | Im u].
// isB = 1: complex row c = 2 I + m (m = 0 S, 1 H) -> real rows 2c =
// [Re v | Im v] and 2c+1 = [-Im v | Re v], so that a real dot product with
// [Re u | Im u] gives Re and Im of u conj(v).  out: [S][L][rows][Kp] int8,
// Kp = 2 Kcp; ex: [L][complex rows] exponents.  32 complex rows per block.
template <int S>
// A non-finite operand value sets L1G_STATUS_NONFINITE in status (int8
// slices cannot carry it into the products).
__global__ void __launch_bounds__(256, 2) k_sph_slice(DevProb P, const SphCoef* __restrict__ coef, int isB, int Kcp,
                                                      int ncrow, int8_t* __restrict__ out, int* __restrict__ ex,
                                                      int* __restrict__ status) {
  extern __shared__ double2 tile[];  // [Kc][33]
  __shared__ double red[8][32];
  __shared__ int rexp[32];
  const int l = blockIdx.y, L = P.ltop;
  const int rc0 = blockIdx.x * 32;
  const int tid = threadIdx.x;
  const int Kc = 2 * P.ndf, Kp = 2 * Kcp;
  const int nrow_real = isB ? 2 * ncrow : ncrow;  // real rows per l
  // values: one (row, atom) per thread and pass, AL/BL and the phase read
  // once for the atom's two k (and, for B, for both the S and H rows of I)
  const int nrr = isB ? 16 : 32;  // distinct basis rows of the block
  for (int idx = tid; idx < nrr * P.ndf; idx += 256) {
    const int rr = idx % nrr, a = idx / nrr;
    const int row = isB ? (rc0 >> 1) + rr : rc0 + rr;  // J or I
    double al = 0.0, bl = 0.0;
    double2 ph = make_double2(0.0, 0.0);
    const int t = P.atype[a];
    if (row < P.nv) {
      const size_t o = ((size_t)t * L + l) * P.nvpad + row;
      al = P.al[o];
      bl = P.bl[o];
      ph = P.phase[(size_t)a * P.npad + row];
    }
    if (!isB) {
      const bool in = rc0 + rr < ncrow;
      tile[(2 * a) * 33 + rr] = in ? make_double2(ph.x * al, ph.y * al) : make_double2(0.0, 0.0);
      tile[(2 * a + 1) * 33 + rr] = in ? make_double2(ph.x * bl, ph.y * bl) : make_double2(0.0, 0.0);
    } else {
      const SphCoef c = coef[t * L + l];
      const double xs0 = c.vif * al, xs1 = c.vif * (c.chn * bl);                                  // S row
      const double xh0 = c.vif * (c.mAA * al + c.mAB * bl), xh1 = c.vif * (c.mBA * al + c.mBB * bl);  // H row
      const bool in0 = rc0 + 2 * rr < ncrow, in1 = rc0 + 2 * rr + 1 < ncrow;
      tile[(2 * a) * 33 + 2 * rr] = in0 ? make_double2(ph.x * xs0, ph.y * xs0) : make_double2(0.0, 0.0);
      tile[(2 * a + 1) * 33 + 2 * rr] = in0 ? make_double2(ph.x * xs1, ph.y * xs1) : make_double2(0.0, 0.0);
      tile[(2 * a) * 33 + 2 * rr + 1] = in1 ? make_double2(ph.x * xh0, ph.y * xh0) : make_double2(0.0, 0.0);
      tile[(2 * a + 1) * 33 + 2 * rr + 1] = in1 ? make_double2(ph.x * xh1, ph.y * xh1) : make_double2(0.0, 0.0);
    }
  }
  __syncthreads();
  {
    bool bad = false;
    for (int idx = tid; idx < 32 * Kc; idx += 256) bad |= l1g_nonfinite(tile[(idx >> 5) * 33 + (idx & 31)]);
    if (bad) atomicOr(status, L1G_STATUS_NONFINITE);
  }
  {
    const int r = tid & 31, part = tid >> 5;
    double m = 0.0;
    for (int k = part; k < Kc; k += 8) {
      const double2 v = tile[k * 33 + r];
      m = fmax(m, fmax(fabs(v.x), fabs(v.y)));
    }
    red[part][r] = m;
    __syncthreads();
    if (tid < 32) {
      double mm = 0.0;
      for (int q = 0; q < 8; q++) mm = fmax(mm, red[q][tid]);
      const int e = (mm > 0.0) ? ilogb(mm) + 1 : 0;
      rexp[tid] = e;
      if (rc0 + tid < ncrow) ex[(size_t)l * ncrow + rc0 + tid] = e;
    }
    __syncthreads();
  }
  // one element per thread and pass, lanes along k: conflict-free tile
  // reads (stride 33) and byte stores coalesced along each row
  const size_t plane = (size_t)L * nrow_real * Kp;  // one slice plane
  int8_t* lbase = out + (size_t)l * nrow_real * Kp;
  for (int idx = tid; idx < 32 * Kcp; idx += 256) {
    const int rr = idx / Kcp, k = idx - rr * Kcp;
    const int rc = rc0 + rr;
    if (rc >= ncrow) continue;
    const int e = rexp[rr];
    const double2 v = (k < Kc) ? tile[k * 33 + rr] : make_double2(0.0, 0.0);
    double tr = digit_scale(v.x, e), ti = digit_scale(v.y, e);
#pragma unroll
    for (int p = 0; p < S; p++) {
      const int8_t ar = (int8_t)digit7(tr), ai = (int8_t)digit7(ti);
      int8_t* base = lbase + (size_t)p * plane;
      if (!isB) {
        base[(size_t)rc * Kp + k] = ar;
        base[(size_t)rc * Kp + Kcp + k] = ai;
      } else {
        base[(size_t)(2 * rc) * Kp + k] = ar;
        base[(size_t)(2 * rc) * Kp + Kcp + k] = ai;
        base[(size_t)(2 * rc + 1) * Kp + k] = (int8_t)(-ai);
        base[(size_t)(2 * rc + 1) * Kp + Kcp + k] = ar;
      }
    }
  }
}

// 2^e as a double from its exponent bits: exact for -1022 <= e <= 1023,
// 0 below that range and infinity above it (no branch)
__device__ __forceinline__ double pow2i(int e) {
  return __hiloint2double((min(max(e, -1023), 1024) + 1023) << 20, 0);  // biased exponent 0: the double 0
}

// w = (2l+1) P_l(x) of N pairs from the explicit polynomials: independent
// chains with the coefficients as constant operands, and no values of the
// orders below l to keep.  line: bits of the pairs along one line, which take
// x P_(l-1) at every order (hamilt.F:250-281), so x^l.
template <int N>
__device__ __forceinline__ void leg_weights(int l, const double (&x)[N], unsigned line, double (&w)[N]) {
  switch (l) {
    case 0: leg_poly<0>(x, w); break;
    case 1: leg_poly<1>(x, w); break;
    case 2: leg_poly<2>(x, w); break;
    case 3: leg_poly<3>(x, w); break;
    case 4: leg_poly<4>(x, w); break;
    case 5: leg_poly<5>(x, w); break;
    case 6: leg_poly<6>(x, w); break;
    case 7: leg_poly<7>(x, w); break;
    case 8: leg_poly<8>(x, w); break;
    case 9: leg_poly<9>(x, w); break;
    case 10: leg_poly<10>(x, w); break;
    case 11: leg_poly<11>(x, w); break;
    default: leg_poly<12>(x, w); break;
  }
  static_assert(SPH_LMAX == 13, "one case per order");
  if (line) {
#pragma unroll
    for (int u = 0; u < N; u++)
      if ((line >> u) & 1) {
        double p = (double)(2 * l + 1);
        for (int k = 0; k < l; k++) p *= x[u];
        w[u] = p;
      }
  }
}
// (l-1)/l of the Legendre recursion
struct LegRatio {
  double c[SPH_LMAX];
};
constexpr LegRatio leg_ratio_make() {
  LegRatio r{};
  for (int l = 1; l < SPH_LMAX; l++) r.c[l] = (double)(l - 1) / (double)l;
  return r;
}
__constant__ LegRatio leg_ratio = leg_ratio_make();

// Level sum of one accumulator column, sum_d c_d 2^(-7d), in one of three
// exact forms (LS, chosen on the host from the bound on |c_d|):
//   LS = 2: levels paired in int32 (c_d 128 + c_(d+1)), the pairs combined
//           in int64 into V = sum_d c_d 2^(7(S-1-d)), |V| < 2^51, and V
//           converted by one add (returns V: the caller's scale carries
//           2^(-7(S-1)));
//   LS = 1: pairs in int32, each pair converted and accumulated in FP64;
//   LS = 0: every level converted and accumulated in FP64.
template <int S, int LS>
__device__ __forceinline__ double level_sum(const uint32_t (&r)[S]) {
  if (LS == 2) {
    long long V = 0;
#pragma unroll
    for (int d = 0; d < S; d += 2) {
      if (d + 1 < S)
        V = V * 16384 + (long long)((int)r[d] * 128 + (int)r[d + 1]);
      else
        V = V * 128 + (long long)(int)r[d];
    }
    // 1.5 2^52 + V has V in its low mantissa bits for |V| < 2^51
    return __longlong_as_double(V + 0x4338000000000000LL) - 6755399441055744.0;
  }
  double v = 0.0, w = 1.0;
  if (LS == 1) {
#pragma unroll
    for (int d = 0; d < S; d += 2) {
      if (d + 1 < S) {
        const int pr = (int)r[d] * 128 + (int)r[d + 1];
        v = fma(i2d_exact((uint32_t)pr), w * 0.0078125, v);
      } else {
        v = fma(i2d_exact(r[d]), w, v);
      }
      w *= 6.103515625e-05;  // 2^-14
    }
  } else {
#pragma unroll
    for (int d = 0; d < S; d++) {
      v = fma(i2d_exact(r[d]), w, v);
      w *= 0.0078125;
    }
  }
  return v;
}

// S levels x 4 columns of this warp's TMEM lanes into registers (async until
// tmem_wait4)
template <int S>
__device__ __forceinline__ void tmem_ld4(uint32_t (&r)[S][4], uint32_t addr, int N) {
#pragma unroll
  for (int d = 0; d < S; d++)
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[d][0]), "=r"(r[d][1]), "=r"(r[d][2]), "=r"(r[d][3])
                 : "r"(addr + (uint32_t)(d * N)));
}
// wait for this thread's TMEM loads; the registers pass through an empty asm
// so that no use of them is scheduled before the wait
template <int S>
__device__ __forceinline__ void tmem_wait4(uint32_t (&r)[S][4]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int d = 0; d < S; d++) asm volatile("" : "+r"(r[d][0]), "+r"(r[d][1]), "+r"(r[d][2]), "+r"(r[d][3]));
}
// a table load issued where it stands (volatile: not sunk below the stores)
__device__ __forceinline__ double2 ld_table(const double2* p) {
  double2 v;
  asm volatile("ld.global.nc.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}
// bounded wait that also gives up once another role has raised the abort flag
__device__ __forceinline__ bool wait_or_abort(uint64_t* bar, uint32_t parity, const int* flag) {
  long long t0 = clock64();
  while (!mbar_try_wait(bar, parity))
    if (*(volatile const int*)flag || clock64() - t0 > (1LL << 31)) return false;
  return true;
}

// test hook: a wait on a barrier that nothing arrives at, with a short bound
// (about half a millisecond): false, and the caller takes its timeout path (the
// other roles' waits keep their full bound)
__device__ __forceinline__ bool never_arrives(uint64_t* bar) {
  const long long t0 = clock64();
  bool in_time = true;
  while (in_time && !mbar_try_wait(bar, 0)) in_time = clock64() - t0 <= (1LL << 20);
  return in_time;
}

// Position in a ring of N slots: the slot and the parity of the current
// round's completion (counters and divisions would cost the issuing warps
// more than an MMA)
template <int N>
struct Ring {
  int slot = 0;
  uint32_t par = 0;
  __device__ __forceinline__ void next() {
    if (++slot == N) {
      slot = 0;
      par ^= 1;
    }
  }
};

// Persistent: CTA b takes tiles b, b + gridDim.x, ... of the list.  The
// stage ring and the two accumulator buffers run on counters that continue
// across tiles, so the loads and MMAs of a tile's first l overlap the
// previous tile's last epilogue, interstitial gather and HS writes.
template <int S, int LS, int KB>
__global__ void __launch_bounds__(Cfg<S, KB>::THREADS, 1)
    k_sph_tc(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, DevProb P,
             const int2* __restrict__ tiles, int ntile, int nkb, int klast, int npA, int npB,
             const int* __restrict__ exA, const int* __restrict__ exB, const double2* __restrict__ tab, TabDesc T,
             double2* __restrict__ hs, int ld, double2* __restrict__ hsdiag, int* __restrict__ status,
             int never_wait) {
  using C = Cfg<S, KB>;
  constexpr int N = C::N, IT = C::IT, STAGES = C::STAGES, IPT = C::IPT, EPI = C::EPI;
  constexpr int MMA_WARP = 4 * C::EG, TMA_WARP = 4 * C::EG + 1;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full[STAGES], empty[STAGES], tfull[2], tempty[2], accbar, ebar, never;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // warp-uniform to the compiler
  const int L = P.ltop, nv = P.nv;

  if (warp == MMA_WARP) {
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
    for (int b = 0; b < 2; b++) {
      mbar_init(&tfull[b], 1);
      mbar_init(&tempty[b], 4 * C::EG);  // one arrival per epilogue warp
    }
    mbar_init(&accbar, 1);
    mbar_init(&ebar, EPI);  // the epilogue threads' barrier (bounded waits)
    mbar_init(&never, 1);   // nothing arrives here (the never_wait test hook)
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;

  if (warp == TMA_WARP) {
    // ---- TMA producer: a full ring ahead of the MMAs ----
    if (lane == 0) {
      // a stage of the ring's first round is free, a later one once its last
      // round's MMAs have completed (n: stages issued, up to a full ring)
      Ring<STAGES> r;
      int n = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < ntile && ok; t += gridDim.x) {
        const int2 tt = tiles[t];
        const int j0 = tt.x * 128, i0 = tt.y * IT;
        for (int l = 0; l < L && ok; l++)
          for (int kb = 0; kb < nkb; kb++) {
            if (n == STAGES && !wait_or_abort(&empty[r.slot], r.par ^ 1, &abort_flag)) {
              ok = false;
              break;
            }
            uint8_t* a = smem + r.slot * C::STAGE;
            mbar_expect_tx(&full[r.slot], C::STAGE);
            tma_load_3d(a, &tmA, &full[r.slot], kb * KB, l * npA + j0, 0);
            tma_load_3d(a + C::A_BYTES, &tmB, &full[r.slot], kb * KB, l * 4 * npB + 4 * i0, 0);
            r.next();
            if (n < STAGES) n++;
          }
      }
      if (!ok) atomicOr(status, L1G_STATUS_TIMEOUT);
      // the copies in flight land before the CTA's shared memory is released
      // (the MMA issuer may stop early; consumed stages return at once)
      for (int q = 0; q < n; q++) {  // each stage's last round: this one below the position, else the one before
        const int st = (r.slot + STAGES - 1 - q) % STAGES;
        mbar_wait(&full[st], st < r.slot ? r.par : r.par ^ 1);
      }
    }
    __syncwarp();
  } else if (warp == MMA_WARP) {
    // ---- MMA issuer: the whole warp walks the loop (uniform operands stay
    // in uniform registers), one elected lane issues.  Issued from a branch
    // of one lane instead, each MMA took about 110 clocks of that lane, more
    // than its 77 clocks on the tensor core.
    {
      Ring<STAGES> r;
      Ring<2> rt;     // accumulator buffers, one per l in turn
      int fresh = 2;  // of them not yet used once
      bool ok = true;
      // warp-uniform outcome
      auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
        return __all_sync(0xffffffffu, wait_or_abort(bar, parity, &abort_flag));
      };
      if (never_wait) ok = __all_sync(0xffffffffu, never_arrives(&never));
      const uint64_t desc0 = desc_kblock<KB>(smem_u32(smem));
      for (int t = blockIdx.x; t < ntile && ok; t += gridDim.x) {
        for (int l = 0; l < L && ok; l++) {
          if (fresh > 0)
            fresh--;
          else
            ok = wait(&tempty[rt.slot], rt.par ^ 1);
          for (int kb = 0; kb < nkb && ok; kb++) {
            ok = wait(&full[r.slot], r.par);
            if (!ok) break;
            tc_fence_after();
            const uint64_t ad0 = desc0 + (uint32_t)(r.slot * (C::STAGE >> 4)), bd0 = ad0 + (C::A_BYTES >> 4);
            const uint32_t d0 = tmem + (uint32_t)(rt.slot * S * N);
            // the last block holds klast valid 32-byte steps (TMA zero-fills
            // the rest; their MMAs are skipped)
            const int nh = (kb == nkb - 1) ? klast : C::KSTEPS;
            if (elect_one()) {
              // The S slices of B lie one after another in shared memory (one
              // (S N)-row K-major tile) and the level accumulators N columns
              // apart in TMEM, so A slice p times B slices 0..S-1-p is ONE MMA
              // of width (S-p) N whose columns land on levels p..S-1
#pragma unroll
              for (int k = 0; k < C::KSTEPS; k++)
                if (k < nh) {
#pragma unroll
                  for (int p = 0; p < S; p++)
                    mma_i8(d0 + p * N, ad0 + ((p * 128 * KB + k * 32) >> 4), bd0 + ((k * 32) >> 4),
                           idesc_i8(128, (S - p) * N), (k > 0 || p > 0) ? 1u : (uint32_t)(kb > 0));
                }
              mma_commit(&empty[r.slot]);
              if (kb == nkb - 1) mma_commit(&tfull[rt.slot]);
            }
            __syncwarp();
            r.next();
          }
          rt.next();
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
    // ---- epilogue warps ----
    double* sU = (double*)(smem + STAGES * C::STAGE);  // [IT][4]: k_I / |k_I| (0 for a zero row) and |k_I|
    int* sK = (int*)(sU + 4 * IT);                   // [IT][4]: KZZ
    int16_t* sA = (int16_t*)(sK + 4 * IT);            // [l][128]: eA - 12
    int16_t* sB = sA + SPH_LMAX * 128;                    // [l][IT][2]: eB
    const int g4 = warp & 3, hh = warp >> 2;
    // Up to 5 slices the Legendre weights come from the polynomials, with x
    // from the rows' unit vectors: the recursion's x and two last values per
    // pair would take 6 registers each.  6 and 7 slices keep the recursion
    // (its rounding is the reference's).
    constexpr bool POLY = S <= 5;
    const uint32_t trow = tmem + ((uint32_t)(32 * g4) << 16);
    Ring<2> rt;  // as the MMA issuer's
    bool ok = true;
    uint32_t ephase = 0;
    // barrier of the epilogue threads on an mbarrier, every wait bounded
    // (a warp that gave up leaves the others to time out, not to hang);
    // warp-uniform outcome
    auto epi_sync = [&]() -> bool {
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&ebar)) : "memory");
      const bool r = __all_sync(0xffffffffu, wait_or_abort(&ebar, ephase & 1, &abort_flag));
      ephase++;
      return r;
    };
    // this thread's share of a tile's scale tables, fetched into registers
    // one tile ahead (behind the previous tile's interstitial part)
    constexpr int QA = (SPH_LMAX * 128 + EPI - 1) / EPI, QB = (SPH_LMAX * 2 * IT + EPI - 1) / EPI;
    int16_t pa[QA], pb[QB];
    int2 tn = make_int2(0, 0);          // the next tile
    auto fetch = [&](int t) {  // volatile loads: issued here, ahead of their use
      tn = make_int2(split::ld_early(&tiles[t].x), split::ld_early(&tiles[t].y));
      const int j0 = tn.x * 128, i0 = tn.y * IT;
#pragma unroll
      for (int k = 0; k < QA; k++) {
        const int q = tid + k * EPI, l = q >> 7, J = j0 + (q & 127);
        pa[k] = (int16_t)((q < L * 128 && J < nv) ? split::ld_early(&exA[(size_t)l * npA + J]) - 12
                                                   : -2000);  // -2000: a zero scale
      }
#pragma unroll
      for (int k = 0; k < QB; k++) {
        const int q = tid + k * EPI, l = q / (2 * IT), r = q % (2 * IT), I = i0 + (r >> 1);
        pb[k] = (int16_t)((q < L * 2 * IT && I < nv) ? split::ld_early(&exB[(size_t)l * 2 * npB + 2 * I + (r & 1)])
                                                      : -2000);
      }
    };
    if (blockIdx.x < ntile) fetch(blockIdx.x);
    for (int t = blockIdx.x; t < ntile; t += gridDim.x) {
      const int j0 = tn.x * 128, i0 = tn.y * IT;
      // this thread's J row, and one I row per thread of the first warps
      const int J = j0 + 32 * g4 + lane;
      const bool jin = J < nv;
      const int Jr = min(J, nv - 1), Ir = min(i0 + tid, nv - 1);
      const double rj = P.rk[Jr], vj = rj > 0.0 ? 1.0 / rj : 0.0;
      const double ux = P.xk[Jr] * vj, uy = P.yk[Jr] * vj, uz = P.zk[Jr] * vj;
      const int k1 = P.kzz[3 * Jr], k2 = P.kzz[3 * Jr + 1], k3 = P.kzz[3 * Jr + 2];
      double ri = 0.0, xi = 0.0, yi = 0.0, zi = 0.0;
      int ki1 = 0, ki2 = 0, ki3 = 0;
      if (tid < IT) {
        ri = P.rk[Ir];
        const double vi = ri > 0.0 ? 1.0 / ri : 0.0;
        xi = P.xk[Ir] * vi;
        yi = P.yk[Ir] * vi;
        zi = P.zk[Ir] * vi;
        ki1 = P.kzz[3 * Ir];
        ki2 = P.kzz[3 * Ir + 1];
        ki3 = P.kzz[3 * Ir + 2];
      }
      // row and scale tables of this tile, written once the previous
      // tile's readers are past the first barrier
      if (!epi_sync()) {
        ok = false;
        break;
      }
#pragma unroll
      for (int k = 0; k < QA; k++)
        if (tid + k * EPI < L * 128) sA[tid + k * EPI] = pa[k];
#pragma unroll
      for (int k = 0; k < QB; k++)
        if (tid + k * EPI < L * 2 * IT) sB[tid + k * EPI] = pb[k];
      if (tid < IT) {
        sU[4 * tid] = xi;
        sU[4 * tid + 1] = yi;
        sU[4 * tid + 2] = zi;
        sU[4 * tid + 3] = ri;
        sK[4 * tid] = ki1;
        sK[4 * tid + 1] = ki2;
        sK[4 * tid + 2] = ki3;
      }
      if (!epi_sync()) {
        ok = false;
        break;
      }
      // cosine of the pair's k vectors (li: I within the tile)
      auto cosine = [&](int li) { return fma(ux, sU[4 * li], fma(uy, sU[4 * li + 1], uz * sU[4 * li + 2])); };
      double x[POLY ? 1 : IPT], pm1[POLY ? 1 : IPT], pm2[POLY ? 1 : IPT];
      double2 aS[IPT], aH[IPT];
      unsigned top = 0, flat = 0;  // pairs along one line (hamilt.F's UTOP branch); pairs with a (nearly) zero row
#pragma unroll
      for (int u = 0; u < IPT; u++) {
        const int li = hh * IPT + u;
        double xx = 0.0;
        if (jin && i0 + li < nv) {
          xx = cosine(li);
          const double den = rj * sU[4 * li + 3];
          if (!(den > 1.0e-8)) {  // the reference's x is k_J.k_I itself: at most 1e-8
            flat |= 1u << u;
            xx *= den;
          }
        }
        if (!(fabs(xx) < 0.9999999)) top |= 1u << u;
        if (!POLY) {
          x[u] = xx;
          pm1[u] = xx;   // P_1
          pm2[u] = 1.0;  // P_0
        }
        aS[u] = aH[u] = make_double2(0.0, 0.0);
      }
      for (int l = 0; l < L; l++, rt.next()) {
        const int buf = rt.slot;
        // scales (2l+1) P_l 2^(eA + eB) of this thread's pairs: formed
        // before the wait, which hides them when the MMAs are behind
        const int ea = sA[l * 128 + 32 * g4 + lane] + (LS == 2 ? -7 * (S - 1) : 0);
        double sS[IPT], sH[IPT];
        {
          double w[IPT];
          if (POLY) {
            double xx[IPT];
#pragma unroll
            for (int u = 0; u < IPT; u++) {
              xx[u] = cosine(hh * IPT + u);
              if ((flat >> u) & 1) xx[u] = 0.0;
            }
            leg_weights(l, xx, top, w);
          } else {
            // Legendre recursion (hamilt.F:250-281, UTOP branch)
            const double cl = leg_ratio.c[l], fl = (double)(2 * l + 1);
#pragma unroll
            for (int u = 0; u < IPT; u++) {
              double pl;
              if (l == 0)
                pl = 1.0;
              else if (l == 1)
                pl = x[u];
              else {
                if (!((top >> u) & 1)) {
                  const double pplx = x[u] * pm1[u];
                  pl = pplx + cl * (pplx - pm2[u]);
                } else {
                  pl = x[u] * pm1[u];
                }
                pm2[u] = pm1[u];
                pm1[u] = pl;
              }
              w[u] = fl * pl;
            }
          }
#pragma unroll
          for (int u = 0; u < IPT; u++) {
            const short2 sb = *reinterpret_cast<const short2*>(sB + (l * IT + hh * IPT + u) * 2);
            sS[u] = w[u] * pow2i(ea + sb.x);
            sH[u] = w[u] * pow2i(ea + sb.y);
          }
        }
        // warp-uniform outcome: the TMEM loads below are .sync.aligned
        if (!__all_sync(0xffffffffu, wait_or_abort(&tfull[buf], rt.par, &abort_flag))) {
          ok = false;
          if (lane == 0) atomicOr(status, L1G_STATUS_TIMEOUT);
          break;
        }
        if (__any_sync(0xffffffffu, *(volatile int*)&abort_flag)) {
          ok = false;
          break;
        }
        tc_fence_after();
        // 4 real columns per I: S re, S im, H re, H im; this thread's I start
        // at column 4 IPT hh; one I (4 columns x S levels) per load
        const uint32_t tcol = trow + (uint32_t)(buf * S * N + 4 * IPT * hh);
#pragma unroll
        for (int u = 0; u < IPT; u++) {
          uint32_t r[S][4];
          tmem_ld4<S>(r, tcol + 4 * u, N);
          tmem_wait4<S>(r);
          if (u == IPT - 1) {
            // all columns of this buffer read: hand it back to the MMA issuer
            tc_fence_before();
            __syncwarp();
            if (lane == 0)
              asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&tempty[buf])) : "memory");
          }
          double v[4];
#pragma unroll
          for (int m = 0; m < 4; m++) {
            uint32_t rr[S];
#pragma unroll
            for (int d = 0; d < S; d++) rr[d] = r[d][m];
            v[m] = level_sum<S, LS>(rr);
          }
          aS[u].x = fma(v[0], sS[u], aS[u].x);
          aS[u].y = fma(v[1], sS[u], aS[u].y);
          aH[u].x = fma(v[2], sH[u], aH[u].x);
          aH[u].y = fma(v[3], sH[u], aH[u].y);
        }
      }
      if (!ok) {
        *(volatile int*)&abort_flag = 1;
        break;
      }
      if (t + (int)gridDim.x < ntile) fetch(t + gridDim.x);
      // interstitial + write (hamilt.F:289-345, 459-466, calkpt.F:164)
      if (jin) {
        const int nx = 2 * T.d1 + 1, ny = 2 * T.d2 + 1;
        // table values of NG pairs at a time, the next NG in flight while
        // these are written; I past NV reads a valid entry and stores nothing
        constexpr int NG = 2;
        double2 th[2][NG], wp[2][NG];
        auto gather = [&](int g, double2(&a)[NG], double2(&b)[NG]) {
#pragma unroll
          for (int w = 0; w < NG; w++) {
            const int li = hh * IPT + g * NG + w;
            const int d1 = k1 - sK[4 * li] + T.d1, d2 = k2 - sK[4 * li + 1] + T.d2, d3 = k3 - sK[4 * li + 2] + T.d3;
            const size_t ci = ((size_t)d3 * ny + d2) * nx + d1;
            a[w] = ld_table(tab + 2 * ci);
            b[w] = ld_table(tab + 2 * ci + 1);
          }
        };
        bool bad = false;  // a written element is not finite
        gather(0, th[0], wp[0]);
#pragma unroll
        for (int g = 0; g < IPT / NG; g++) {
          if (g + 1 < IPT / NG) gather(g + 1, th[(g + 1) & 1], wp[(g + 1) & 1]);
#pragma unroll
          for (int w = 0; w < NG; w++) {
            const int u = g * NG + w, li = hh * IPT + u, I = i0 + li;
            if (I >= nv || J > I) continue;
            const double x2 = cosine(li) * (rj * sU[4 * li + 3]);
            const double2 s = cadd(th[g & 1][w], aS[u]);
            const double2 hv = cadd(cadd(cscale(th[g & 1][w], x2), wp[g & 1][w]), aH[u]);
            if (J == I) {
              hs[(size_t)I * ld + I] = hv;
              hsdiag[I] = s;
            } else {
              hs[(size_t)I * ld + J] = s;   // S upper: HS(J,I)
              hs[(size_t)J * ld + I] = hv;  // H lower: HS(I,J)
            }
            bad |= l1g_nonfinite(s) | l1g_nonfinite(hv);
          }
        }
        if (bad) atomicOr(status, L1G_STATUS_NONFINITE);
      }
    }
    if (!ok) {
      *(volatile int*)&abort_flag = 1;
      if (lane == 0) atomicOr(status, L1G_STATUS_TIMEOUT);
    }
  }
  // every MMA issued has completed before TMEM is freed
  if (warp == MMA_WARP) mbar_wait(&accbar, 0);
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

}  // namespace sphtc
