// dmb_oz64.cu -- products of complex128 matrices on the INT8 tensor cores, to
// FP64 accuracy: the trailing updates of the complex128 LDL^T
//
//   F(m, j) -= sum_k W(m, k) L(j, k),  j <= m  (row-major F, W, L).
//
// The residue scheme of dmb_ozaki.cu with both operands FP64: row m of W and
// row j of L are scaled by powers of two and rounded to 55-bit integers (one
// bit below the rounding of an FP64 value of the row's largest exponent), the
// integer product is formed modulo 16 coprime moduli (M ~ 2^125.4 >
// 2 K 2^110 for K = 2 x 1024) by exact int8 products, and recombined as a
// 96-bit fraction.  The only errors are the two roundings to 55 bits and one
// rounding of the result; an FP64 sum of K products rounds K times.
//
// The roundings are relative to the largest element of a row, so the columns
// are balanced first: column k of W = L D is scaled by 2^-e, column k of L by
// 2^e, 4^e about |D_k| (exact).  Both rows are then rows of about L sqrt(|D|),
// whose elements do not carry the scales of the basis functions of their
// columns.  Without it the error grew with the spread of these scales.  Largest
// |A - L D L^T| over the diagonal scales, updates of 64 columns emulated on the
// host, plates of 519 unknowns with graded cells: scales over 1.6e3 2e-11, balanced
// 1e-13, FP64 sums 1e-13; over 3e6 0.4, 3e-9 and 2e-9; even plates and disks 1e-15 to
// 3e-15 in all three.
//
// Why: B200 has no FP64 tcgen05 kind, and an FP64-pipe GEMM stops at 36.8
// TFLOP/s (a complex MAC = 8 flops); 16 int8 products at the nominal int8
// rate amount to 280.  Measured (trailing updates of a 7,680-unknown factor):
// 4.0 us per modulus and 64 x 128 x 1,024 tile and SM, 155 TFLOP/s, against 18
// for the FP64-pipe kernel (37 sustained by cuBLAS); bound by the operand
// feed from L2 (96 KB a us and SM) for K = 1,024, by the drain (1.85 us a
// unit) for K = 256.
//
// Three launches per update:
//  k_oz64_planes  both operands' scales and residues.  Complex row r of an
//                 operand takes two int8 rows of K bytes, 32 (r / 16) + r % 16
//                 (real parts) and 16 further (imaginary parts), so the same
//                 planes serve as A and as B.
//  k_oz64_gemm    persistent; a unit is one modulus of one 64 x 128 complex
//                 tile: one M 128, N 256 int8 product whose accumulator holds,
//                 for 16 rows and 16 columns at a time, the four products
//                 rr, ri / ir, ii of real and imaginary parts.  Lane l of a
//                 warp (real row) and lane l + 16 (imaginary row) exchange
//                 their products with the imaginary columns, so each forms its
//                 part of the complex product, reduces it and stores one byte.
//                 Units are independent, so they go round-robin over the CTAs
//                 (modulus by modulus: one modulus' planes stay in L2), and an
//                 update of a few tiles still occupies every SM.
//  k_oz64_crt     the 16 residues of each element to FP64, subtracted from F
//                 in coalesced 64-byte pieces, at full occupancy: 26 us for a
//                 7,424 x 256 update.  (As the last drain of the product's own
//                 eight warps, exposed to L2 latency, it took 85 us.)
#include <algorithm>
#include <cmath>

#include "dmb_device.cuh"
#include "dmb_internal.h"
#include "dmb_residue.cuh"

namespace {

using namespace dmb_tc;

constexpr int O6_STAGES = 4;
constexpr int O6_A_STAGE = OZ_BM * OZ_BK, O6_B_STAGE = OZ_BN * OZ_BK;
constexpr int O6_SMEM = O6_STAGES * (O6_A_STAGE + O6_B_STAGE) + 256 /*barriers*/ + 1024 /*align*/;
constexpr int O6_DRAIN = 16;                         // drain warps
constexpr int O6_THREADS = 32 * (O6_DRAIN + 2);      // and the TMA producer and the MMA issuer
constexpr int O6_BM = 64, O6_BN = 128;               // complex tile
constexpr int O6_RES_PLANE = 2 * O6_BM * O6_BN;      // residues of one unit
constexpr int64_t O6_RES_TILE = (int64_t)OZ_NMOD64 * O6_RES_PLANE;
constexpr int O6_BITS = 55;   // |scaled integer| <= 2^55
constexpr int O6_SHIFT = 50;  // row scales are kept as 2^(e - O6_SHIFT): finite for every finite row

struct Sched64 {
  int mod[OZ_NMOD64];
  unsigned mmul[OZ_NMOD64], moff[OZ_NMOD64];             // oz_mod
  unsigned f0[OZ_NMOD64], f1[OZ_NMOD64], f2[OZ_NMOD64];  // round(2^96 y_i / m_i), 32 bits each
  double cscale;                                         // M 2^-64 2^(-2 bits) 2^(2 O6_SHIFT)
};

// Tiles of the lower part of an update whose rows start 128 d below its
// columns, column tile by column tile: column tile ct has the row tiles from
// 2 (ct - d) on.
struct Tiles64 {
  int nrt, ncol;
  int64_t d;
  __host__ __device__ int first(int ct) const {
    const int64_t f = 2 * (ct - d);
    return (int)(f < 0 ? 0 : f > nrt ? nrt : f);
  }
  __host__ __device__ void at(int64_t t, int &rt, int &ct) const {
    for (ct = 0; ct < ncol - 1; ct++) {
      const int n = nrt - first(ct);
      if (t < n) break;
      t -= n;
    }
    rt = first(ct) + (int)t;
  }
  int64_t count() const {
    int64_t n = 0;
    for (int ct = 0; ct < ncol; ct++) n += nrt - first(ct);
    return n;
  }
};

__global__ void __launch_bounds__(O6_THREADS, 1) k_oz64_gemm(const __grid_constant__ CUtensorMap tmA,
                                                             const __grid_constant__ CUtensorMap tmB,
                                                             const __grid_constant__ Sched64 sc, int kchunks,
                                                             Tiles64 tl, int64_t ntiles, int arow, int brow,
                                                             unsigned char *__restrict__ Rres, unsigned *err) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char *gbase = smem_raw + (base - raw);
  const uint32_t sA = base;
  const uint32_t sB = base + O6_STAGES * O6_A_STAGE;
  const uint32_t sBar = sB + O6_STAGES * O6_B_STAGE;
  uint64_t *bar_ptr = reinterpret_cast<uint64_t *>(gbase + (sBar - base));
  volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(bar_ptr + 16);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(bar_ptr + 17);
  const uint32_t full0 = sBar, empty0 = sBar + 8 * O6_STAGES, accf0 = sBar + 16 * O6_STAGES, acce0 = accf0 + 16,
                 fin = acce0 + 16;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < O6_STAGES; s++) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int b = 0; b < 2; b++) {
      mbar_init(accf0 + 8 * b, 1);
      mbar_init(acce0 + 8 * b, O6_DRAIN);  // one arrival per drain warp
    }
    mbar_init(fin, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(const_cast<uint32_t *>(tmem_slot))),
                 "r"(2 * OZ_BN)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_d = *tmem_slot;
  const int64_t units = ntiles * OZ_NMOD64;

  if (warp == O6_DRAIN) {
    if (lane == 0) {
      long long t = 0;
      bool go = true;
      for (int64_t u = blockIdx.x; go && u < units; u += gridDim.x) {
        const int i = (int)(u / ntiles);
        int rt, ct;
        tl.at(u - i * ntiles, rt, ct);
        for (int kc = 0; kc < kchunks; kc++, t++) {
          const int s = (int)(t % O6_STAGES);
          if (*abort_flag ||
              (t >= O6_STAGES && !mbar_wait(empty0 + 8 * s, (uint32_t)((t / O6_STAGES) - 1) & 1u, err, abort_flag))) {
            go = false;
            break;
          }
          mbar_expect_tx(full0 + 8 * s, O6_A_STAGE + O6_B_STAGE);
          tma_load_2d(sA + s * O6_A_STAGE, &tmA, kc * OZ_BK, i * arow + OZ_BM * rt, full0 + 8 * s);
          tma_load_2d(sB + s * O6_B_STAGE, &tmB, kc * OZ_BK, i * brow + OZ_BN * ct, full0 + 8 * s);
        }
      }
      // given up: the last fill of each stage
      for (long long f = t > O6_STAGES ? t - O6_STAGES : 0; !go && f < t; f++)
        mbar_wait_in_flight(full0 + 8 * (int)(f % O6_STAGES), (uint32_t)(f / O6_STAGES) & 1u);
    }
  } else if (warp == O6_DRAIN + 1) {
    if (lane == 0) {
      long long t = 0;
      int g = 0;
      bool ok = true;
      for (int64_t u = blockIdx.x; ok && u < units; u += gridDim.x, g++) {
        // unit g accumulates in buffer g & 1, free once unit g - 2 drained
        if (g >= 2 && !mbar_wait(acce0 + 8 * (g & 1), (uint32_t)((g >> 1) - 1) & 1u, err, abort_flag)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t acc = tmem_d + (uint32_t)((g & 1) * OZ_BN);
        for (int kc = 0; kc < kchunks; kc++, t++) {
          const int s = (int)(t % O6_STAGES);
          if (!mbar_wait(full0 + 8 * s, (uint32_t)(t / O6_STAGES) & 1u, err, abort_flag)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
          for (int k = 0; k < OZ_BK / 32; k++)
            umma_i8(acc, sw128_desc(sA + s * O6_A_STAGE + k * 32), sw128_desc(sB + s * O6_B_STAGE + k * 32),
                    (kc == 0 && k == 0) ? 0u : 1u);
          umma_commit(empty0 + 8 * s);
        }
        if (ok) umma_commit(accf0 + 8 * (g & 1));
      }
      if (!ok) {  // given up: the products issued
        umma_commit(fin);
        mbar_wait_in_flight(fin, 0);
      }
    }
  } else {
    // each drain warp works alone on the 32 TMEM lanes of its quarter (warp &
    // 3) and on a quarter of the columns (warp >> 2): groups of 16 real and 16
    // imaginary columns; element q of a group goes to byte q / 4 of word q % 4
    // (a lane of k_oz64_crt then holds columns 4 apart, four lanes 64 bytes of F)
    const int row = (warp & 3) * 32 + lane;
    const bool im = lane >= 16;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    int g = 0;
    for (int64_t u = blockIdx.x; u < units; u += gridDim.x, g++) {
      const int i = (int)(u / ntiles);
      const int64_t tile = u - i * ntiles;
      uint4 *Rt = reinterpret_cast<uint4 *>(Rres + tile * O6_RES_TILE + (int64_t)i * O6_RES_PLANE) + row;
      const unsigned gm = (unsigned)sc.mod[i], gmul = sc.mmul[i], goff = sc.moff[i];
      const bool got = mbar_wait(accf0 + 8 * (g & 1), (uint32_t)(g >> 1) & 1u, err, abort_flag);
      if (!__all_sync(0xffffffffu, got)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t tacc = tmem_d + (uint32_t)((g & 1) * OZ_BN) + lane_base;
#pragma unroll
      for (int x = 0; x < 32 / O6_DRAIN; x++) {
        const int cc = (warp >> 2) * (32 / O6_DRAIN) + x;
        uint32_t v[32];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
            "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
              "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
              "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]),
              "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]),
              "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
            : "r"(tacc + (uint32_t)(cc * 32)));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        unsigned w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int q = 0; q < 16; q++) {
          // real lane: Sr Lr - Si Li, imaginary lane: Si Lr + Sr Li
          const int o = __shfl_xor_sync(0xffffffffu, (int)v[16 + q], 16);
          w[q & 3] |= oz_mod((int)v[q] + (im ? o : -o), gm, gmul, goff) << (8 * (q >> 2));
        }
        Rt[cc * 128] = make_uint4(w[0], w[1], w[2], w[3]);
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(acce0 + 8 * (g & 1));
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "r"(2 * OZ_BN) : "memory");
}

// F -= the product whose residues Rres holds: CTA (tile, 16-column group), a
// thread for 4 columns (4 apart) of one row; rows M x columns C of F at (m0,
// c0) of an update whose row and column 0 coincide.  sum_i r_i f_i mod 2^96
// is kept in three 32-bit columns (16 terms of 8 x 32 bits stay below 2^44).
__global__ void __launch_bounds__(256) k_oz64_crt(const __grid_constant__ Sched64 sc, Tiles64 tl, int64_t M, int64_t C,
                                                  int64_t m0, int64_t c0, const double *__restrict__ rs,
                                                  const double *__restrict__ cs, double2 *__restrict__ F, int64_t ldf,
                                                  const unsigned char *__restrict__ Rres) {
  const int64_t tile = blockIdx.x >> 3;
  const int grp = blockIdx.x & 7, l4 = threadIdx.x & 3, crow = threadIdx.x >> 2;
  int rt, ct;
  tl.at(tile, rt, ct);
  const int64_t m = (int64_t)O6_BM * rt + crow, cb = (int64_t)O6_BN * ct + 16 * grp + l4;
  if (m >= M) return;
  const int64_t c_end = min(C, m0 + m + 1 - c0);  // below the diagonal and inside the update
  if (cb >= c_end) return;
  const unsigned *R = reinterpret_cast<const unsigned *>(Rres + tile * O6_RES_TILE) +
                      4 * (grp * 128 + 32 * (crow >> 4) + (crow & 15)) + l4;
  unsigned w[2][OZ_NMOD64];
#pragma unroll
  for (int j = 0; j < OZ_NMOD64; j++) {
    w[0][j] = R[j * (O6_RES_PLANE / 4)];
    w[1][j] = R[j * (O6_RES_PLANE / 4) + 64];
  }
  double2 *Fp = F + m * ldf + cb;
  double2 f[4];
  double s[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const bool in = cb + 4 * q < c_end;
    f[q] = in ? Fp[4 * q] : make_double2(0, 0);
    s[q] = in ? cs[cb + 4 * q] : 0.0;
  }
  const double rsc = rs[m] * sc.cscale;
#pragma unroll
  for (int p = 0; p < 2; p++) {
    unsigned long long a0[4], a1[4];
    unsigned a2[4];
#pragma unroll
    for (int q = 0; q < 4; q++) a0[q] = a1[q] = a2[q] = 0;
#pragma unroll
    for (int j = 0; j < OZ_NMOD64; j++)
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const unsigned u = (w[p][j] >> (8 * q)) & 0xffu;
        a0[q] += (unsigned long long)u * sc.f0[j];
        a1[q] += (unsigned long long)u * sc.f1[j];
        a2[q] += u * sc.f2[j];
      }
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const unsigned long long hi = ((unsigned long long)a2[q] << 32) + a1[q] + (a0[q] >> 32);
      const double x = fma((double)(unsigned)a0[q], 0x1p-32, (double)(long long)hi) * (rsc * s[q]);
      if (p == 0) f[q].x -= x;
      else f[q].y -= x;
    }
  }
#pragma unroll
  for (int q = 0; q < 4; q++)
    if (cb + 4 * q < c_end) Fp[4 * q] = f[q];
}

// constants of the residues of a 57-bit integer given as bytes: weights 256^j
// mod m (j = 0..7) for two dp4a, the bias that undoes u = x + 2^56 and centres
// the residue, the reciprocal ceil(2^32 / m)
struct Mods64 {
  unsigned wlo[OZ_NMOD64], whi[OZ_NMOD64], bias[OZ_NMOD64], mul[OZ_NMOD64];
  int m[OZ_NMOD64], half[OZ_NMOD64];
};

struct Operand64 {
  const double2 *S;   // rows x K, row-major
  int64_t ld, rows, padded;
  const short *bal;   // exponents of the K columns, and their sign for this operand
  int sign;
  double *scale;      // padded
  signed char *P;     // OZ_NMOD64 planes of 2 padded rows of K bytes
};

// Residue planes and scales of both operands; rows from `rows` to `padded` are
// zero.  1024 / K rows per CTA, staged through shared memory (a thread
// handles 16 consecutive values so that its residues leave as 16-byte stores;
// one value of padding per 16 keeps its reads free of bank conflicts).
// Integer arithmetic: per value and modulus two dp4a on the bytes of the
// 57-bit integer, one multiply-high, one multiply-add (the FP64 reduction of
// k_oz_res_a takes a rounding, a fused multiply-add, two comparisons and a
// conversion on slower pipes).  A row with a non-finite value gets the scale
// NaN, so that the update carries it on as the FP64 product would.
template <int K>
__global__ void __launch_bounds__(64) k_oz64_planes(Operand64 A, Operand64 B, const __grid_constant__ Mods64 md) {
  constexpr int RPB = 1024 / K, TPR = K / 16;  // rows per CTA, threads per row
  __shared__ double2 st[1024 + 64];
  __shared__ double red[2];
  __shared__ int bad[RPB];
  const int64_t na = A.padded / RPB;
  const Operand64 &O = blockIdx.x < na ? A : B;
  const int64_t r0 = (int64_t)(blockIdx.x < na ? blockIdx.x : blockIdx.x - na) * RPB;
  const int t = threadIdx.x, rl = t / TPR, kt = t % TPR;
  const int64_t r = r0 + rl;
  if (t < RPB) bad[t] = 0;
#pragma unroll
  for (int u = 0; u < 16; u++) {
    const int e = t + 64 * u;
    const int64_t rr = r0 + e / K;
    st[e + (e >> 4)] = rr < O.rows ? O.S[rr * O.ld + e % K] : make_double2(0, 0);
  }
  // this thread's columns: exponents two to a word, |e| < 540
  const uint4 b0 = reinterpret_cast<const uint4 *>(O.bal + 16 * kt)[0], b1 = reinterpret_cast<const uint4 *>(O.bal + 16 * kt)[1];
  const unsigned be[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
  __syncthreads();
  const double2 *my = st + 17 * t;
  auto value = [&](int u) {  // balanced: times 2^(sign e), exact
    const int e = (short)(u & 1 ? be[u >> 1] >> 16 : be[u >> 1] & 0xffffu);
    return cscale(my[u], __hiloint2double((1023 + O.sign * e) << 20, 0));
  };
  double mx = 0.0;
  bool finite = true;
#pragma unroll
  for (int u = 0; u < 16; u++) {
    const double2 v = value(u);
    mx = fmax(mx, fmax(fabs(v.x), fabs(v.y)));
    finite = finite && isfinite(v.x) && isfinite(v.y);
  }
  if (!finite) bad[rl] = 1;
#pragma unroll
  for (int o = (TPR < 32 ? TPR : 32) / 2; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (TPR > 32 && (t & 31) == 0) red[t >> 5] = mx;
  __syncthreads();
  if (TPR > 32) mx = fmax(red[0], red[1]);
  const bool nan = bad[rl] != 0;
  int e = 0;
  if (mx > 0.0 && !nan) frexp(mx, &e);
  e = max(e, -900);  // smaller rows than 2^-900: products of them round to nothing
  if (kt == 0) O.scale[r] = nan ? __longlong_as_double(0x7ff8000000000000ll) : ldexp(1.0, e - O6_SHIFT);
  const double f = ldexp(1.0, O6_BITS - e);
  const int64_t row = 32 * (r / 16) + r % 16;
  signed char *Pr = O.P + row * K + 16 * kt;
#pragma unroll
  for (int c = 0; c < 2; c++) {
    unsigned lo[16], hi[16];
#pragma unroll
    for (int u = 0; u < 16; u++) {
      const double v = c == 0 ? value(u).x : value(u).y;
      const unsigned long long a = (unsigned long long)(__double2ll_rn(nan ? 0.0 : v * f) + (1ll << 56));
      lo[u] = (unsigned)a;
      hi[u] = (unsigned)(a >> 32);
    }
#pragma unroll 4
    for (int i = 0; i < OZ_NMOD64; i++) {
      unsigned w[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        unsigned b[4];
#pragma unroll
        for (int x = 0; x < 4; x++) {
          const unsigned v = __dp4a(lo[4 * q + x], md.wlo[i], __dp4a(hi[4 * q + x], md.whi[i], md.bias[i]));
          // in [-half, m - half): the low byte is the int8 residue
          b[x] = v - __umulhi(v, md.mul[i]) * md.m[i] - md.half[i];
        }
        w[q] = __byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410);
      }
      *reinterpret_cast<uint4 *>(Pr + ((int64_t)i * 2 * O.padded + 16 * c) * K) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

const Mods64 &mods64() {
  static const Mods64 md = [] {
    Mods64 x{};
    for (int i = 0; i < OZ_NMOD64; i++) {
      const unsigned m = (unsigned)OZ_MODULI[i];
      unsigned p = 1 % m, w[8];
      for (int j = 0; j < 8; j++) {
        w[j] = p;
        p = (p * 256u) % m;
      }
      x.wlo[i] = w[0] | (w[1] << 8) | (w[2] << 16) | (w[3] << 24);
      x.whi[i] = w[4] | (w[5] << 8) | (w[6] << 16) | (w[7] << 24);
      x.half[i] = (int)(m / 2);  // residues in [-half, m - half): [-(m-1)/2, (m-1)/2] for odd m, [-128, 127] for 256
      x.bias[i] = (m - w[7]) % m + m / 2;  // 2^56 = 256^7
      x.mul[i] = (unsigned)(((1ull << 32) + m - 1) / m);
      x.m[i] = (int)m;
    }
    return x;
  }();
  return md;
}

const Sched64 &sched64() {
  static const Sched64 sc = [] {
    Sched64 s{};
    const CrtConst k = crt_const(OZ_NMOD64);
    for (int i = 0; i < OZ_NMOD64; i++) {
      s.mod[i] = OZ_MODULI[i];
      s.mmul[i] = (unsigned)((((uint64_t)1 << 39) + OZ_MODULI[i] - 1) / OZ_MODULI[i]);
      s.moff[i] = (unsigned)(OZ_MODULI[i] * ((1u << 31) / OZ_MODULI[i]));
      s.f0[i] = k.fraclo[i];
      s.f1[i] = (unsigned)k.frac[i];
      s.f2[i] = (unsigned)(k.frac[i] >> 32);
    }
    DMB_REQUIRE(crt_fits(2 * 1024, 2 * O6_BITS, k), DMB_ERR_STATE, "int8 residue update: K out of range");
    s.cscale = std::ldexp((double)k.M, -64 - 2 * O6_BITS + 2 * O6_SHIFT);
    return s;
  }();
  return sc;
}

int64_t up(int64_t v, int64_t m) { return ((v + m - 1) / m) * m; }

// Operand and residue planes are made for at most this many rows / columns at
// a time (multiples of 128): 0.8 GB a stream whatever the matrix size.
constexpr int64_t O6_ROWS_1024 = 4096, O6_ROWS_256 = 16384, O6_COLS = 4096;

// A stream's part of the buffer: operand planes, row scales of both operands,
// residue planes of `tiles` tiles, for padded sizes mp x cp
struct Part64 {
  size_t scale, res, end;
  Part64(int64_t mp, int64_t cp, int64_t tiles, int K) {
    scale = up((int64_t)OZ_NMOD64 * 2 * (mp + cp) * K, 1024);
    res = scale + up(sizeof(double) * (mp + cp), 1024);
    end = res + (size_t)tiles * O6_RES_TILE;
  }
};

}  // namespace

namespace dmb {

bool oz64_available(dmb_ctx *c, int K) { return tc_available(c) && (K == 256 || K == 1024); }

// bytes an update of M rows and C columns needs of its stream's part
size_t oz64_bytes(int64_t M, int64_t C, int K) {
  const int64_t mc = up(std::min(M, K == 1024 ? O6_ROWS_1024 : O6_ROWS_256), O6_BM), cc = up(std::min(C, O6_COLS), O6_BN);
  const Tiles64 tl{(int)(mc / O6_BM), (int)(cc / O6_BN), M > mc ? cc / O6_BN : 0};
  return Part64(mc, cc, tl.count(), K).end;
}

// One buffer for a factorisation's three streams and its column exponents: an
// allocation takes 0.33 ms and a release 0.3, whatever their size, so nothing grows on
// the way (nine buffers that did cost the first factorisation of a context 5 ms)
bool oz64_reserve(dmb_ctx *c, int64_t N, const size_t (&bytes)[3]) {
  Oz64State &st = c->oz64;
  size_t at = up(sizeof(short) * N, 1024);
  for (int s = 0; s < 3; s++) {
    st.part[s] = at;
    at += up(bytes[s], 1024);
  }
  try {
    st.buf.ensure(at);
  } catch (const DmbError &) {
    (void)cudaGetLastError();  // no room: the caller keeps to the FP64 pipe
    return false;
  }
  return true;
}

void oz64_lower_update(dmb_ctx *c, int64_t M, int64_t C, int K, const double2 *W, int64_t ldw, const double2 *L,
                       int64_t ldl, const short *bal, double2 *F, int64_t ldf, int slot, unsigned *err) {
  Oz64State &st = c->oz64;
  raise_smem(c, k_oz64_gemm, O6_SMEM);
  const int64_t mstep = K == 1024 ? O6_ROWS_1024 : O6_ROWS_256;
  for (int64_t c0 = 0; c0 < C; c0 += O6_COLS) {
    const int64_t nc = std::min(O6_COLS, C - c0), ncp = up(nc, O6_BN);
    for (int64_t m0 = c0 / mstep * mstep; m0 < M; m0 += mstep) {
      const int64_t nm = std::min(mstep, M - m0), nmp = up(nm, O6_BM);
      const Tiles64 tl{(int)(nmp / O6_BM), (int)(ncp / O6_BN), (m0 - c0) / O6_BN};
      const int64_t ntiles = tl.count();
      if (ntiles == 0) continue;
      const Part64 part(nmp, ncp, ntiles, K);
      char *base = st.buf.as<char>() + st.part[slot];
      double *rs = (double *)(base + part.scale), *cs = rs + nmp;
      signed char *PA = (signed char *)base, *PB = PA + (size_t)OZ_NMOD64 * 2 * nmp * K;
      unsigned char *res = (unsigned char *)(base + part.res);
      const Operand64 A{W + m0 * ldw, ldw, nm, nmp, bal, -1, rs, PA}, B{L + c0 * ldl, ldl, nc, ncp, bal, 1, cs, PB};
      const unsigned g = (unsigned)((nmp + ncp) / (1024 / K));
      if (K == 1024)
        DMB_LAUNCH(c, k_oz64_planes<1024>, g, 64, 0, A, B, mods64());
      else
        DMB_LAUNCH(c, k_oz64_planes<256>, g, 64, 0, A, B, mods64());
      CUtensorMap mA, mB;
      make_map_bytes(&mA, PA, CU_TENSOR_MAP_DATA_TYPE_UINT8, (uint64_t)K, (uint64_t)K, (uint64_t)(OZ_NMOD64 * 2 * nmp),
                     OZ_BK, OZ_BM);
      make_map_bytes(&mB, PB, CU_TENSOR_MAP_DATA_TYPE_UINT8, (uint64_t)K, (uint64_t)K, (uint64_t)(OZ_NMOD64 * 2 * ncp),
                     OZ_BK, OZ_BN);
      const int64_t G = std::min<int64_t>(ntiles * OZ_NMOD64, c->sm_count);
      DMB_LAUNCH(c, k_oz64_gemm, (unsigned)G, O6_THREADS, O6_SMEM, mA, mB, sched64(), K / OZ_BK, tl, ntiles,
                 (int)(2 * nmp), (int)(2 * ncp), res, err);
      DMB_LAUNCH(c, k_oz64_crt, (unsigned)(ntiles * 8), 256, 0, sched64(), tl, nm, nc, m0, c0, (const double *)rs,
                 (const double *)cs, F + m0 * ldf + c0, ldf, res);
    }
  }
}

void oz64_release(dmb_ctx *c) { c->oz64.buf.release(); }

}  // namespace dmb
