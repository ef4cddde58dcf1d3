// dmb_factor.cu -- near-field preconditioner: extraction, factorisation, apply.
//
//   * extraction (NearFieldPreconditioner.jl:247-369, 429-464, 670-716):
//     Z_nf[m][n] = Z[m][n] when the RWG centres are within `cutoff`
//     (inclusive, exact tie-break), else 0; nnz counted for nnz_ratio.
//   * Jacobi (:623-668): 1 / z_ii with the 1e-10 * max|z_ii| floor.
//   * factorisation: Z_nf is complex symmetric (Z is, and the distance test is
//     symmetric), so it is factored as L D L^T -- unit lower L, diagonal D, no
//     pivoting -- which has the same inverse as the reference's UMFPACK LU up to
//     rounding, at half the flops.  Right-looking, panel width NB = 64:
//       k_ldlt_mid     a 256-wide panel (four diagonal blocks, their panel rows
//                      and the updates between them) in one launch;
//     and updates A22 -= (L21 D1) L21^T after every 256 and 1,024 columns
//     (complex128: int8 residue products, dmb_oz64.cu, or the FP64 pipe;
//     complex64: the tensor-core kernels of dmb_tc.cu or FP32 units).
//     A zero or non-finite pivot stops with DMB_ERR_BREAKDOWN.
//   * apply (NearFieldOperator, :1034-1054): L y = x, z = y / D, L^T x = z; up
//     to seven columns by one data-flow launch per sweep (k_sweep_fwd /
//     k_sweep_bwd, 256-row blocks and their inverses), more columns by panels.
//     Every wait is bounded: on expiry the kernel sets an error bit and returns;
//     the host raises DMB_ERR_TIMEOUT.
#include <algorithm>
#include <type_traits>
#include <cmath>
#include <cstring>

#include "dmb_device.cuh"
#include "dmb_internal.h"

namespace dmb {
void tc_ldlt_update_c64(dmb_ctx *c, int64_t N, int64_t r0, int64_t c_hi, int64_t jcol, int K, float2 *F,
                        const float2 *W, int wstride, int woff, int slot);
}  // namespace dmb

namespace {

constexpr int NB = 64;  // panel width == triangular-solve block

unsigned blocks_for(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

// ---------------------------------------------------------------------------
// near-field extraction
// ---------------------------------------------------------------------------
__device__ bool within_cutoff_exact(const double *a, const double *b, double cutoff) {
  // compare the exact squared distance with cutoff^2 in double-double
  double s = 0, e = 0;
  double v[3] = {a[0] - b[0], a[1] - b[1], a[2] - b[2]};
  for (int i = 0; i < 3; i++) {
    double p = v[i] * v[i], pe = fma(v[i], v[i], -p);
    double t = s + p, bb = t - s;
    e += (s - (t - bb)) + (p - bb) + pe;
    s = t;
  }
  double c2 = cutoff * cutoff, c2e = fma(cutoff, cutoff, -c2);
  return (s - c2) + (e - c2e) <= 0.0;
}

// 32 x 32 tiles; centres staged in shared memory; the squared distance is
// compared with a band around cutoff^2 and only the band goes to the exact test
template <class ZC, class FC>
__global__ void __launch_bounds__(256) k_nf_mask(int64_t N, const ZC *__restrict__ Z, const double *__restrict__ cen,
                                                 double cutoff, FC *__restrict__ F,
                                                 unsigned long long *__restrict__ nnz) {
  __shared__ double cm[32][3], cn[32][3];
  int64_t m0 = (int64_t)blockIdx.y * 32, n0 = (int64_t)blockIdx.x * 32;
  int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  if (threadIdx.x < 96) {
    int i = threadIdx.x / 3, d = threadIdx.x % 3;
    cm[i][d] = (m0 + i < N) ? cen[3 * (m0 + i) + d] : 0.0;
    cn[i][d] = (n0 + i < N) ? cen[3 * (n0 + i) + d] : 0.0;
  }
  __syncthreads();
  const bool all_in = !isfinite(cutoff);
  const double c2 = cutoff * cutoff;
  const double lo = c2 * (1 - 1e-12), hi = c2 * (1 + 1e-12);
  unsigned keep_cnt = 0;
  int64_t n = n0 + tx;
  for (int i = ty; i < 32; i += 8) {
    int64_t m = m0 + i;
    if (m >= N || n >= N) continue;
    bool keep;
    if (all_in) keep = true;
    else if (cutoff <= 0.0) keep = (m == n);
    else {
      double dx = cm[i][0] - cn[tx][0], dy = cm[i][1] - cn[tx][1], dz = cm[i][2] - cn[tx][2];
      double d2 = dx * dx + dy * dy + dz * dz;
      keep = (m == n) || d2 < lo || (d2 <= hi && within_cutoff_exact(cm[i], cn[tx], cutoff));
    }
    store_c(F + m * N + n, keep ? to_d2(Z[m * N + n]) : make_double2(0, 0));
    keep_cnt += keep;
  }
  unsigned cnt = __reduce_add_sync(0xffffffffu, keep_cnt);
  if ((threadIdx.x & 31) == 0 && cnt) atomicAdd(nnz, (unsigned long long)cnt);
}

template <class ZC>
__global__ void k_diag_max(int64_t N, const ZC *__restrict__ Z, double *__restrict__ out, unsigned *__restrict__ bad) {
  __shared__ double red[32];
  double mx = 0;
  for (int64_t i = threadIdx.x; i < N; i += blockDim.x) {
    double2 z = to_d2(Z[i * N + i]);
    double a = hypot(z.x, z.y);
    if (!isfinite(a)) atomicOr(bad, 1u);
    mx = fmax(mx, a);
  }
  mx = warp_max(mx);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x / 32] = mx;
  __syncthreads();
  if (threadIdx.x < 32) {
    mx = threadIdx.x < blockDim.x / 32 ? red[threadIdx.x] : 0;
    mx = warp_max(mx);
    if (threadIdx.x == 0) *out = mx;
  }
}

template <class ZC>
__global__ void k_diag_inv(int64_t N, const ZC *__restrict__ Z, const double *__restrict__ maxabs,
                           double2 *__restrict__ dinv) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  double floor_abs = 1e-10 * (*maxabs);
  if (floor_abs == 0.0) floor_abs = 4.9406564584124654e-324;
  double2 z = to_d2(Z[i * N + i]);
  if (hypot(z.x, z.y) < floor_abs) z = make_double2(floor_abs, 0);
  dinv[i] = cdiv(make_double2(1, 0), z);
}

// ---------------------------------------------------------------------------
// LDL^T kernels; C is the storage and compute type (double2 or float2)
// ---------------------------------------------------------------------------
// 1 / x for a positive normal float: the hardware approximation refined by
// one Newton-Raphson step, r <- r (2 - x r)
__device__ __forceinline__ float rcp_nr(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r * fmaf(-x, r, 2.f);
}
// the same for doubles: two Newton-Raphson steps
__device__ __forceinline__ double rcp_nr(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  r = fma(r, fma(-x, r, 1.0), r);
  return fma(r, fma(-x, r, 1.0), r);
}
// 1 / d of a pivot: conj(d) / |d|^2; FP64 pivots whose |d|^2 leaves the
// normal range are divided by Smith's algorithm
__device__ __forceinline__ float2 pivot_inverse(float2 d) {
  const float rd = rcp_nr(fmaf(d.x, d.x, d.y * d.y));
  return make_float2(d.x * rd, -d.y * rd);
}
__device__ __forceinline__ double2 pivot_inverse(double2 d) {
  const double d2 = fma(d.x, d.x, d.y * d.y);
  if (d2 > 1e-290 && d2 < 1e290) {
    const double rd = rcp_nr(d2);
    return make_double2(d.x * rd, -d.y * rd);
  }
  return cdiv(make_double2(1.0, 0.0), d);
}
__device__ __forceinline__ float2 cneg(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ double2 cneg(double2 a) { return make_double2(-a.x, -a.y); }

// The plain form for complex128 blocks with a pivot outside the range of the
// fast one below: entry by entry in shared memory, pivots divided by Smith's
// algorithm.  A zero or non-finite pivot is a breakdown.
__device__ __noinline__ bool elim16_any(double2 (*A)[68], double2 (*Xs)[17], int s0, int lane, double2 *dinv) {
  for (int e = lane; e < 256; e += 32) Xs[e >> 4][e & 15] = make_double2((e >> 4) == (e & 15) ? 1.0 : 0.0, 0.0);
  __syncwarp();
  for (int k = 0; k < 16; k++) {
    const double2 d = A[s0 + k][s0 + k];
    const double ad = cabsv(d);
    if (!(ad > 0.0) || !isfinite(ad)) return false;
    const double2 inv_d = cdiv(make_double2(1.0, 0.0), d);
    double2 v[8], x[8];
#pragma unroll
    for (int m = 0; m < 8; m++) {
      const int e = lane + 32 * m, i = e >> 4, c = e & 15;
      const double2 l = cmul(A[s0 + i][s0 + k], inv_d);
      v[m] = c == k ? l : csub(A[s0 + i][s0 + c], cmul(l, A[s0 + c][s0 + k]));
      x[m] = csub(Xs[i][c], cmul(l, Xs[k][c]));
    }
    __syncwarp();
#pragma unroll
    for (int m = 0; m < 8; m++) {
      const int e = lane + 32 * m, i = e >> 4, c = e & 15;
      if (i <= k) continue;
      if (c >= k && c <= i) A[s0 + i][s0 + c] = v[m];
      Xs[i][c] = x[m];
    }
    if (lane == 0) dinv[k] = inv_d;
    __syncwarp();
  }
  return true;
}

// two values at an address that is a multiple of their size
__device__ __forceinline__ void load_pair(const double2 *p, double2 &a, double2 &b) {
  a = p[0];
  b = p[1];
}
__device__ __forceinline__ void load_pair(const float2 *p, float2 &a, float2 &b) {
  const float4 v = *reinterpret_cast<const float4 *>(p);
  a = make_float2(v.x, v.y);
  b = make_float2(v.z, v.w);
}
__device__ __forceinline__ void store_pair(double2 *p, double2 a, double2 b) {
  p[0] = a;
  p[1] = b;
}
__device__ __forceinline__ void store_pair(float2 *p, float2 a, float2 b) {
  *reinterpret_cast<float4 *>(p) = make_float4(a.x, a.y, b.x, b.y);
}

// Elimination of the 16 x 16 diagonal sub-block at s0 by one warp, the values
// in registers: lane c < 16 holds column c of the upper triangle (the block is
// complex symmetric), lane 16 + c column c of the unit-lower inverse X.  Row k,
// which by symmetry is also the column of multipliers, goes to all lanes through
// shared memory, two rows at a time (buf: two pairs of 32 values in turn); then
// every lane takes the same steps, t = a_k / d, a_i -= a_ki t for i > k, without
// a select or a branch: entries below the diagonal are garbage that nobody
// reads, and the rows of X are subject to the same operations.  Unrolled, so that the registers
// are named at compile time.  Bound by the chain rows -> two reciprocals ->
// update -> next rows of a single warp: 5,300 cycles a block (complex128 7,900)
// against 30,000 with a lane holding eight entries of a column, whose selects
// and predicated exchange stores came to 1,900 cycles a pivot, and 10,400 with
// one row an exchange.  On return the lower triangle holds L (strict) and
// D, Xs the unit-lower inverse, dinv the reciprocal pivots.  Complex64: a pivot
// whose |d|^2 is zero, non-finite or outside the FP32 normal range (|d| below
// ~1e-19 or above ~1e19) is a breakdown; complex128 ones outside the fast range
// go to elim16_any.
template <class C, int LD>
__device__ __forceinline__ bool elim16_warp(C (*A)[LD], C (*Xs)[17], int s0, int lane, C *buf, C *dinv) {
  constexpr bool f64 = sizeof(C) == 16;
  const int c = lane & 15;
  const bool isx = lane >= 16;
  C a[16];
#pragma unroll
  for (int i = 0; i < 16; i++) {
    const C v = A[s0 + c][s0 + (i <= c ? i : 0)];
    a[i] = isx ? (i == c ? cone<C>() : czero<C>()) : i <= c ? v : czero<C>();
  }
  bool ok = true;
  auto invert = [&](C d) {
    if constexpr (f64) {
      const double d2 = fma(d.x, d.x, d.y * d.y);
      ok = ok && d2 > 1e-290 && d2 < 1e290;
      const double rd = rcp_nr(d2);
      return make_double2(d.x * rd, -d.y * rd);
    } else {
      const float d2 = fmaf(d.x, d.x, d.y * d.y);
      ok = ok && d2 >= 1.17549435e-38f && d2 <= 3.40282347e38f;
      const float rd = rcp_nr(d2);
      return make_float2(d.x * rd, -d.y * rd);
    }
  };
#pragma unroll
  for (int k = 0; k < 16; k += 2) {
    C *row = buf + 64 * ((k >> 1) & 1);
    store_pair(row + 2 * lane, a[k], a[k + 1]);
    __syncwarp();
    // r_i = row[2 i], s_i = row[2 i + 1]: rows k and k + 1 before this step
    C d0, r1, d1;
    d0 = row[2 * k];
    load_pair(row + 2 * k + 2, r1, d1);
    const C inv0 = invert(d0), l = cmul(r1, inv0);
    cfma(d1, cneg(r1), l);
    const C inv1 = invert(d1);
    if (lane == 0) {
      dinv[k] = inv0;
      dinv[k + 1] = inv1;
    }
    C t0 = cneg(cmul(a[k], inv0));
    cfma(a[k + 1], r1, t0);
    const C t1 = cneg(cmul(a[k + 1], inv1));
    cfma(t0, cneg(l), t1);  // r_i t0 + (s_i - l r_i) t1 = r_i (t0 - l t1) + s_i t1
#pragma unroll
    for (int i = k + 2; i < 16; i++) {
      C r, s;
      load_pair(row + 2 * i, r, s);
      cfma(a[i], r, t0);
      cfma(a[i], s, t1);
    }
  }
  if (!__all_sync(0xffffffffu, ok)) {
    if constexpr (f64) return elim16_any(A, Xs, s0, lane, dinv);
    return false;
  }
  __syncwarp();  // dinv
#pragma unroll
  for (int i = 0; i < 16; i++) {
    if (isx) Xs[i][c] = a[i];
    else if (i <= c) A[s0 + c][s0 + i] = i < c ? cmul(a[i], dinv[i]) : a[i];
  }
  return true;
}

// Shared memory of a diagonal tile's factorisation: the tile A, the sub-panel
// Wp, the inverses Xd of its 16 x 16 diagonal blocks, its inverse LI.  The
// leading dimension of complex128 tiles suits the FP64 matrix instruction's
// fragments (8 rows x 4 columns of 16 bytes without bank conflicts).
template <class C> struct DiagSmem {
  static constexpr int LD = sizeof(C) == 16 ? 68 : 65;
  static constexpr size_t bytes = sizeof(C) * (2 * 64 * LD + 64 * 17 + 4 * 16 * 17 + 32) + 16;
  C (*A)[LD];
  C (*Wp)[17];
  C (*Xd)[16][17];
  C (*LI)[LD];
  C *dinv;
  int *bad;
  __device__ explicit DiagSmem(unsigned char *smem) {
    C *p = reinterpret_cast<C *>(smem);
    A = reinterpret_cast<C(*)[LD]>(p);
    Wp = reinterpret_cast<C(*)[17]>(p + 64 * LD);
    Xd = reinterpret_cast<C(*)[16][17]>(p + 64 * LD + 64 * 17);
    LI = reinterpret_cast<C(*)[LD]>(p + 64 * LD + 64 * 17 + 4 * 16 * 17);
    dinv = p + 2 * 64 * LD + 64 * 17 + 4 * 16 * 17;
    bad = reinterpret_cast<int *>(dinv + 32);
  }
};

// Blocked factorisation of a 64 x 64 diagonal tile: four 16-wide sub-panels.
// Warp 0 eliminates the 16 x 16 diagonal sub-block in registers (elim16_warp,
// which also forms its unit-lower inverse X), the CTA forms W = A21 X^T below
// it, and warp 0 updates the next diagonal sub-block and goes on with it while
// the other warps store L21 = W D^-1 and update the rest; the products are
// 8 x 8 tiles of FP64 matrix instructions for both types (complex64 on FP32 units
// took twice as long).  Rows and columns at or beyond b are padded with the
// identity (D = 1, L = 0).
// Phase 1 of the blocked factorisation: L and D of the diagonal tile (in
// shared memory: lower triangle, identity padding; written back to F) and the
// unit-lower inverses Xd of its four 16 x 16 diagonal blocks.  Returns false
// after a breakdown (uniform).
template <class C>
__device__ bool ldlt_diag_phase1(int64_t N, int64_t j, int b, C *__restrict__ F, unsigned *__restrict__ err,
                                 unsigned char *smem) {
  DiagSmem<C> sm(smem);
  auto A = sm.A;
  auto Wp = sm.Wp;
  auto Xd = sm.Xd;
  C *dinv = sm.dinv;
  volatile int *bad = sm.bad;
  const int t = threadIdx.x;  // 256 threads
  if (t == 0) *bad = 0;
  __syncthreads();
  const int warp = t >> 5, l4 = t & 3, l8 = (t & 31) >> 2;
  for (int s = 0;; s++) {
    const int s0 = 16 * s;
    if (s > 0) {
      // the step below sub-panel s - 1, whose W has nr rows from s0
      const int nr = 64 - s0, nt = nr / 8 * (nr / 8 + 1) / 2;
      const C *dv = dinv + 16 * ((s - 1) & 1);
      // tile q of the lower tiles of A22 (row by row) -= W (W D^-1)^T
      auto update = [&](int q) {
        int ti = 0, tj = q;
        while (tj > ti) tj -= ++ti;
        const int r = s0 + 8 * ti, cc = s0 + 8 * tj;
        double ur[2] = {0.0, 0.0}, ui[2] = {0.0, 0.0};
#pragma unroll
        for (int k = 0; k < 16; k += 4)
          zmma(ur, ui, to_d2(Wp[r + l8][k + l4]), to_d2(cmul(Wp[cc + l8][k + l4], dv[k + l4])));
#pragma unroll
        for (int u = 0; u < 2; u++) {
          C &v = A[r + l8][cc + 2 * l4 + u];
          store_c(&v, csub(to_d2(v), make_double2(ur[u], ui[u])));
        }
      };
      if (warp != 0)
        for (int e = t - 32; e < nr * 16; e += 224) {
          const int r = s0 + (e >> 4), c = e & 15;
          const C l = cmul(Wp[r][c], dv[c]);
          A[r][s0 - 16 + c] = l;
          if (r < b && s0 - 16 + c < b) F[(j + r) * N + j + s0 - 16 + c] = l;
        }
#pragma unroll 1
      for (int q = warp == 0 ? 0 : 2 + warp; q < (warp == 0 ? 3 : nt); q += warp == 0 ? 1 : 7) update(q);
    }
    if (warp == 0) {
      __syncwarp();
      // its exchange rows in Wp are above those of W
      if (!elim16_warp(A, Xd[s], s0, t, &Wp[0][0], dinv + 16 * (s & 1)) && t == 0) {
        atomicOr(err, 2u);
        *bad = 1;
      }
    }
    __syncthreads();
    if (*bad) return false;  // uniform
    if (s == 3) break;
    // W = A21 X^T: 12, 8 or 4 tiles, a warp takes every eighth
    for (int q = warp; q < 2 * (6 - 2 * s); q += 8) {
      const int r = s0 + 16 + 8 * (q >> 1), cj = 8 * (q & 1);
      double wr[2] = {0.0, 0.0}, wi[2] = {0.0, 0.0};
#pragma unroll
      for (int k = 0; k < 16; k += 4)
        if (k < cj + 8) zmma(wr, wi, to_d2(A[r + l8][s0 + k + l4]), to_d2(Xd[s][cj + l8][k + l4]));
#pragma unroll
      for (int u = 0; u < 2; u++) store_c(&Wp[r + l8][cj + 2 * l4 + u], make_double2(wr[u], wi[u]));
    }
    __syncthreads();
  }
  // the diagonal 16 x 16 blocks
  for (int e = t; e < 4 * 256; e += blockDim.x) {
    const int i = 16 * (e >> 8) + ((e >> 4) & 15), c = 16 * (e >> 8) + (e & 15);
    if (i < b && c <= i) F[(j + i) * N + j + c] = A[i][c];
  }
  return true;
}

// Phase 2: the unit-lower inverse of the factored tile (L in shared memory)
// by recursive doubling from the four 16 x 16 inverses of phase 1, and its
// store to Linv.
template <class C>
__device__ void ldlt_diag_phase2(C *__restrict__ Linv, unsigned char *smem) {
  DiagSmem<C> sm(smem);
  auto A = sm.A;
  auto Wp = sm.Wp;
  auto Xd = sm.Xd;
  auto LI = sm.LI;
  const int t = threadIdx.x;
  // Linv by recursive doubling: 16-level pairs, then the 32-level block
  //   [[X0, 0], [-X1 L10 X0, X1]]
  for (int e = t; e < 64 * 64; e += blockDim.x) {
    const int i = e >> 6, c = e & 63;
    LI[i][c] = ((i >> 4) == (c >> 4)) ? Xd[i >> 4][i & 15][c & 15] : czero<C>();
  }
  // phase A: T_h = L[32h+16.., 32h..] Xd[2h] (two 16 x 16 products, 2 outputs per thread)
  {
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const int e = t + 256 * u, h = e >> 8, r = (e >> 4) & 15, c = e & 15;
      C p0 = czero<C>(), p1 = czero<C>();
#pragma unroll
      for (int k = 0; k < 16; k += 2) {
        cfma(p0, A[32 * h + 16 + r][32 * h + k], Xd[2 * h][k][c]);
        cfma(p1, A[32 * h + 16 + r][32 * h + k + 1], Xd[2 * h][k + 1][c]);
      }
      Wp[32 * h + r][c] = cadd(p0, p1);
    }
  }
  __syncthreads();
  // phase B: LI[32h+16+r][32h+c] = -Xd[2h+1] T_h
  {
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const int e = t + 256 * u, h = e >> 8, r = (e >> 4) & 15, c = e & 15;
      C p0 = czero<C>(), p1 = czero<C>();
#pragma unroll
      for (int k = 0; k < 16; k += 2) {
        if (k <= r) cfma(p0, Xd[2 * h + 1][r][k], Wp[32 * h + k][c]);
        if (k + 1 <= r) cfma(p1, Xd[2 * h + 1][r][k + 1], Wp[32 * h + k + 1][c]);
      }
      const C acc = cadd(p0, p1);
      LI[32 * h + 16 + r][32 * h + c] = cneg(acc);
    }
  }
  __syncthreads();
  // phase C: U = L[32.., 0..32) X_a (32 x 32, X_a lower: k >= c), 4 outputs
  // per thread; U goes to Wp as two 32 x 16 halves (Wp[r][c] for c < 16,
  // Wp[32 + r][c - 16] for c >= 16)
  {
    const int c = t & 31, r0 = t >> 5;  // rows r0, r0 + 8, r0 + 16, r0 + 24
    C p[4] = {czero<C>(), czero<C>(), czero<C>(), czero<C>()};
#pragma unroll
    for (int k = 0; k < 32; k++) {
      if (k >= c) {
        const C x = LI[k][c];
#pragma unroll
        for (int q = 0; q < 4; q++) cfma(p[q], A[32 + r0 + 8 * q][k], x);
      }
    }
    __syncthreads();  // Wp of phase B is consumed
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int r = r0 + 8 * q;
      if (c < 16) Wp[r][c] = p[q];
      else Wp[32 + r][c - 16] = p[q];
    }
  }
  __syncthreads();
  // phase D: LI[32 + r][c] = -X_b U, X_b = LI[32.., 32..] lower (k <= r)
  {
    const int c = t & 31, r0 = t >> 5;
    C p[4] = {czero<C>(), czero<C>(), czero<C>(), czero<C>()};
#pragma unroll
    for (int k = 0; k < 32; k++) {
      const C u = c < 16 ? Wp[k][c] : Wp[32 + k][c - 16];
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (k <= r0 + 8 * q) cfma(p[q], LI[32 + r0 + 8 * q][32 + k], u);
    }
#pragma unroll
    for (int q = 0; q < 4; q++) LI[32 + r0 + 8 * q][c] = cneg(p[q]);
  }
  __syncthreads();
  // (the 16 x 16 diagonal blocks were stored already)
  for (int e = t; e < 64 * 64; e += blockDim.x)
    if ((e >> 10) != ((e & 63) >> 4)) Linv[e] = LI[e >> 6][e & 63];
  __syncthreads();
}

// F[r][c] -= sum_{k<K} W[r][woff+k] F[c][jcol+k] on the 64 x 64 tile at
// (r0, c0), c < c_hi, r >= c, r < N (SIMT; Ws / Ls: 2 x 16 x 65 staging)
template <class C>
__device__ __forceinline__ void ldlt_tile_update(int64_t N, int64_t r0, int64_t c0, int64_t c_hi, int64_t jcol,
                                                 int K, C *__restrict__ F, const C *__restrict__ W, int wstride,
                                                 int woff, C (*Ws)[65], C (*Ls)[65]) {
  int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  C acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int jj = 0; jj < 4; jj++) acc[i][jj] = czero<C>();
  for (int k0 = 0; k0 < K; k0 += 16) {
    for (int e = threadIdx.x; e < 16 * 64; e += 256) {
      int kk = e & 15, rr = e >> 4;
      int64_t r = r0 + rr, cc = c0 + rr;
      bool kin = k0 + kk < K;
      Ws[kk][rr] = (r < N && kin) ? W[r * wstride + woff + k0 + kk] : czero<C>();
      Ls[kk][rr] = (cc < c_hi && kin) ? F[cc * N + jcol + k0 + kk] : czero<C>();
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < 16; kk++) {
      C a[4], l[4];
#pragma unroll
      for (int i = 0; i < 4; i++) a[i] = Ws[kk][ty + 16 * i];
#pragma unroll
      for (int jj = 0; jj < 4; jj++) l[jj] = Ls[kk][tx + 16 * jj];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int jj = 0; jj < 4; jj++) cfma(acc[i][jj], a[i], l[jj]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int jj = 0; jj < 4; jj++) {
      int64_t r = r0 + ty + 16 * i, cc = c0 + tx + 16 * jj;
      if (r < N && cc < c_hi && cc <= r) {
        C *p = F + r * N + cc;
        *p = csub(*p, acc[i][jj]);
      }
    }
}

// Trailing update of a complex64 factor on FP32 units (grid.x row tiles, grid.y
// column tiles from r_lo; tiles entirely above the diagonal exit at once).
template <class C>
__global__ void __launch_bounds__(256) k_ldlt_update(int64_t N, int64_t r_lo, int64_t c_hi, int64_t jcol, int K,
                                                     C *__restrict__ F, const C *__restrict__ W, int wstride,
                                                     int woff) {
  __shared__ C Ws[16][65];
  __shared__ C Ls[16][65];
  const int64_t r0 = r_lo + (int64_t)blockIdx.x * 64, c0 = r_lo + (int64_t)blockIdx.y * 64;
  if (r0 >= N || c0 >= c_hi || c0 > r0 + 63) return;
  ldlt_tile_update<C>(N, r0, c0, c_hi, jcol, K, F, W, wstride, woff, Ws, Ls);
}

// ---------------------------------------------------------------------------
// A 256-wide middle panel in one launch, driven by data flow.  The CTA that
// draws ticket r owns the 64-row tile r (rows J + 64 r ..) of the panel's four
// 64-wide block columns s:
//   * r > s: T = A_rs - sum_{q<s} W_rq L_sq^T as soon as tile s has published
//     its L_sq; then, once tile s has published its factored diagonal block,
//     W_rs L_ss^T = T by forward substitution with the inverses of the 16 x 16
//     blocks (each warp alone on 8 rows), L_rs = W_rs D_s^-1;
//   * r < 4: after each block column its own diagonal tile is updated by
//     W_rs L_rs^T; the last of these updates goes straight to the tile's
//     factorisation (r = s).
// The chain is then, per 64 columns, one factorisation, one substitution and
// one 64 x 64 x 64 update on a single SM; everything else runs while others
// wait.  Tickets are drawn in launch order and a CTA waits only for tiles 0-3,
// which started before it; the waits are bounded (error bit 4).
// The complex128 products are FP64 matrix instructions (mma.sync m8n8k4, full
// FP64 multiply-adds; 37.0 TFLOP/s measured against 33.1 for FMA), which leave
// the shared-memory pipe idle enough to sit at the FP64 rate with eight warps;
// the complex64 ones FP32 FMAs.
// Measured, complex128: 160 us a panel of 1,825 rows (200 us with the block
// elimination on selects and two barriers a pivot; before, a launch with the
// 64-column strip update and the next diagonal block, 105-130 us, and one with
// its panel rows, 17-28 us, per 64 columns).  complex64: 184 us a panel on average
// over a matrix of 4,693 rows with the updates beside it (220 us with the former
// elimination and trailing updates on FP32 units; as much in launches per 64 columns).
// ---------------------------------------------------------------------------
// spin until *flag is set (one thread); false on expiry, this wait's or another
// CTA's (bit 4 of the error word)
__device__ __forceinline__ bool wait_word(volatile unsigned *flag, unsigned *err, long long limit) {
  long long it = 0;
  while (*flag == 0u) {
    if (++it > limit) {
      atomicOr(err, 4u);
      return false;
    }
    if ((it & 255) == 0 && (*(volatile unsigned *)err & 4u)) return false;
    __nanosleep(32);
  }
  __threadfence();
  return true;
}

constexpr int MID_WORDS = 24;  // per middle panel: ticket, diagonal flags [4], row flags [4][4]

// The CTA's share-out of a 64 x 64 product acc += A B^T (A, B rows in shared
// memory, K = 64).  complex128: a warp has 2 x 4 8 x 8 matrix-instruction tiles
// (rows 16 (warp / 2), columns 32 (warp % 2)); complex64: a thread has rows ty +
// 16 i, columns tx + 16 j on FP32 FMAs.  LOWER: only the lower triangle is
// wanted -- complex64 skips the blocks j > i, complex128 deals the 36 lower
// tiles out as warp v < 4: row tile 7 - v, columns 0-4; warp 4 + v: the rest of
// that row tile and row tile v (nine tiles per SM quarter).
template <class C, bool LOWER> struct MidAcc;

template <bool LOWER> struct MidAcc<double2, LOWER> {
  static constexpr int NT = LOWER ? 5 : 8;
  double re[NT][2], im[NT][2];
  int l4, l8, ti[NT], tj[NT], nt;
  __device__ MidAcc() {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    l4 = lane & 3;
    l8 = lane >> 2;
    nt = LOWER && warp >= 4 ? 4 : NT;
#pragma unroll
    for (int x = 0; x < NT; x++) {
      re[x][0] = re[x][1] = im[x][0] = im[x][1] = 0.0;
      const int v = warp & 3;
      if (!LOWER) {
        ti[x] = 2 * (warp >> 1) + x / 4;
        tj[x] = 4 * (warp & 1) + x % 4;
      } else if (warp < 4) {
        ti[x] = 7 - v;
        tj[x] = x;
      } else {
        ti[x] = x < 3 - v ? 7 - v : v;
        tj[x] = x < 3 - v ? 5 + x : x - (3 - v);
      }
    }
  }
  template <int LD> __device__ void mul(const double2 (*A)[LD], const double2 (*B)[LD]) {
    if constexpr (LOWER) {
#pragma unroll 4
      for (int k = 0; k < 64; k += 4)
#pragma unroll
        for (int x = 0; x < NT; x++)
          if (x < nt) zmma(re[x], im[x], A[8 * ti[x] + l8][k + l4], B[8 * tj[x] + l8][k + l4]);
    } else {
#pragma unroll 4
      for (int k = 0; k < 64; k += 4) {
        double2 a[2], b[4];
#pragma unroll
        for (int i = 0; i < 2; i++) a[i] = A[8 * ti[4 * i] + l8][k + l4];
#pragma unroll
        for (int j = 0; j < 4; j++) b[j] = B[8 * tj[j] + l8][k + l4];
#pragma unroll
        for (int x = 0; x < 8; x++) zmma(re[x], im[x], a[x / 4], b[x % 4]);
      }
    }
  }
  // g(row, column, index) for every element; get / set by index
  template <class G> __device__ void each(G g) {
#pragma unroll
    for (int x = 0; x < NT; x++)
      if (x < nt) {
#pragma unroll
        for (int u = 0; u < 2; u++) g(8 * ti[x] + l8, 8 * tj[x] + 2 * l4 + u, 2 * x + u);
      }
  }
  __device__ double2 get(int e) const { return make_double2(re[e >> 1][e & 1], im[e >> 1][e & 1]); }
  __device__ void set(int e, double2 v) {
    re[e >> 1][e & 1] = v.x;
    im[e >> 1][e & 1] = v.y;
  }
};

template <bool LOWER> struct MidAcc<float2, LOWER> {
  float2 acc[4][4];
  int tx, ty;
  __device__ MidAcc() {
    tx = threadIdx.x & 15;
    ty = threadIdx.x >> 4;
#pragma unroll
    for (int e = 0; e < 16; e++) acc[e >> 2][e & 3] = make_float2(0.f, 0.f);
  }
  template <int LD> __device__ void mul(const float2 (*A)[LD], const float2 (*B)[LD]) {
#pragma unroll 8
    for (int k = 0; k < 64; k++) {
      float2 a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; i++) a[i] = A[ty + 16 * i][k];
#pragma unroll
      for (int j = 0; j < 4; j++) b[j] = B[tx + 16 * j][k];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
          if (!LOWER || j <= i) cfma(acc[i][j], a[i], b[j]);
    }
  }
  template <class G> __device__ void each(G g) {
#pragma unroll
    for (int e = 0; e < 16; e++)
      if (!LOWER || (e & 3) <= (e >> 2)) g(ty + 16 * (e >> 2), tx + 16 * (e & 3), e);
  }
  __device__ float2 get(int e) const { return acc[e >> 2][e & 3]; }
  __device__ void set(int e, float2 v) { acc[e >> 2][e & 3] = v; }
};

// W L^T = T in place for the 8 rows Tw of a warp, 16 columns q at a time: T_q -=
// sum_{k < 16 q} W_k L_qk^T, W_q = T_q X_q^T (L: the diagonal tile, X: the
// inverses of its 16 x 16 diagonal blocks); columns at or beyond b are skipped
template <int LD>
__device__ __forceinline__ void mid_substitute(double2 (*Tw)[LD], const double2 (*L)[LD], const double2 (*X)[16][17],
                                               int b) {
  const int lane = threadIdx.x & 31, l4 = lane & 3, l8 = lane >> 2;
#pragma unroll 1
  for (int q = 0; q < 4; q++) {
    if (16 * q >= b) break;  // uniform
    double tr[2][2], ti[2][2];
    if (q > 0) {
#pragma unroll
      for (int n = 0; n < 2; n++)
#pragma unroll
        for (int u = 0; u < 2; u++) {
          const double2 v = Tw[l8][16 * q + 8 * n + 2 * l4 + u];
          tr[n][u] = v.x;
          ti[n][u] = v.y;
        }
      for (int k = 0; k < 16 * q; k += 4) {
        const double2 a = cneg(Tw[l8][k + l4]);
#pragma unroll
        for (int n = 0; n < 2; n++) zmma(tr[n], ti[n], a, L[16 * q + 8 * n + l8][k + l4]);
      }
      __syncwarp();
#pragma unroll
      for (int n = 0; n < 2; n++)
#pragma unroll
        for (int u = 0; u < 2; u++) Tw[l8][16 * q + 8 * n + 2 * l4 + u] = make_double2(tr[n][u], ti[n][u]);
      __syncwarp();
    }
#pragma unroll
    for (int n = 0; n < 2; n++) tr[n][0] = tr[n][1] = ti[n][0] = ti[n][1] = 0.0;
#pragma unroll
    for (int k = 0; k < 16; k += 4) {
      const double2 a = Tw[l8][16 * q + k + l4];
#pragma unroll
      for (int n = 0; n < 2; n++)
        if (k < 8 * n + 8) zmma(tr[n], ti[n], a, X[q][8 * n + l8][k + l4]);
    }
    __syncwarp();
#pragma unroll
    for (int n = 0; n < 2; n++)
#pragma unroll
      for (int u = 0; u < 2; u++) Tw[l8][16 * q + 8 * n + 2 * l4 + u] = make_double2(tr[n][u], ti[n][u]);
    __syncwarp();
  }
}
// complex64: a lane has 2 rows x 2 columns of a step's 8 x 16
template <int LD>
__device__ __forceinline__ void mid_substitute(float2 (*Tw)[LD], const float2 (*L)[LD], const float2 (*X)[16][17],
                                               int b) {
  const int lane = threadIdx.x & 31, r = 2 * (lane >> 3), c = 2 * (lane & 7);
#pragma unroll 1
  for (int q = 0; q < 4; q++) {
    if (16 * q >= b) break;  // uniform
    float2 t[2][2];
#pragma unroll
    for (int u = 0; u < 2; u++)
#pragma unroll
      for (int v = 0; v < 2; v++) t[u][v] = Tw[r + u][16 * q + c + v];
#pragma unroll 8
    for (int k = 0; k < 16 * q; k++) {
      const float2 w0 = cneg(Tw[r][k]), w1 = cneg(Tw[r + 1][k]), l0 = L[16 * q + c][k], l1 = L[16 * q + c + 1][k];
      cfma(t[0][0], w0, l0);
      cfma(t[0][1], w0, l1);
      cfma(t[1][0], w1, l0);
      cfma(t[1][1], w1, l1);
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < 2; u++)
#pragma unroll
      for (int v = 0; v < 2; v++) {
        Tw[r + u][16 * q + c + v] = t[u][v];
        t[u][v] = make_float2(0.f, 0.f);
      }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 16; k++) {  // X is lower triangular with zeros above
      const float2 w0 = Tw[r][16 * q + k], w1 = Tw[r + 1][16 * q + k], x0 = X[q][c][k], x1 = X[q][c + 1][k];
      cfma(t[0][0], w0, x0);
      cfma(t[0][1], w0, x1);
      cfma(t[1][0], w1, x0);
      cfma(t[1][1], w1, x1);
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < 2; u++)
#pragma unroll
      for (int v = 0; v < 2; v++) Tw[r + u][16 * q + c + v] = t[u][v];
    __syncwarp();
  }
}

template <class C>
__global__ void __launch_bounds__(256, sizeof(C) == 16 ? 1 : 2) k_ldlt_mid(int64_t N, int64_t J, int w, C *__restrict__ F,
                                                                           C *__restrict__ Linv, C *__restrict__ W,
                                                                           int wstride, short *__restrict__ bal,
                                                                           unsigned *sync, unsigned *err,
                                                                           long long limit) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned s_ticket;
  __shared__ int s_ok;
  constexpr int LD = DiagSmem<C>::LD;
  DiagSmem<C> sm(smem_raw);
  C(*As)[LD] = sm.A;
  C(*Ls)[LD] = sm.LI;
  C *dinv = &sm.Wp[0][0];  // 64 reciprocal pivots
  unsigned *diag_flag = sync + 1, *row_flag = sync + 5;
  if (threadIdx.x == 0) s_ticket = atomicAdd(sync, 1u);
  __syncthreads();
  const int rt = (int)s_ticket;
  const int t = threadIdx.x, warp = t >> 5;
  const int nsb = (w + 63) / 64;
  const int64_t r0 = J + 64 * (int64_t)rt;
  const int nr = (int)min((int64_t)64, N - r0);
  // wait for a flag, the whole CTA (uniform result)
  auto wait = [&](unsigned *flag) {
    if (t == 0) s_ok = wait_word(flag, err, limit) ? 1 : 0;
    __syncthreads();
    const bool ok = s_ok != 0;
    __syncthreads();
    return ok;
  };
  auto publish = [&](unsigned *flag) {
    __threadfence();
    __syncthreads();
    if (t == 0) atomicExch(flag, 1u);
  };
  // T[64][LD] <- G rows (row r at G + r ld), zero outside nrow x ncol
  auto stage = [&](C(*T)[LD], const C *G, int64_t ld, int nrow, int ncol) {
    C v[16];
#pragma unroll
    for (int m = 0; m < 16; m++) {
      const int e = t + 256 * m, i = e >> 6, c = e & 63;
      v[m] = (i < nrow && c < ncol) ? __ldcg(G + i * ld + c) : czero<C>();
    }
#pragma unroll
    for (int m = 0; m < 16; m++) {
      const int e = t + 256 * m;
      T[e >> 6][e & 63] = v[m];
    }
  };
  for (int s = 0; s < nsb && s <= rt; s++) {
    const int64_t jc = J + 64 * s;
    const int b = (int)min((int64_t)64, J + w - jc);
    if (s == rt) {
      // the diagonal tile (updated by the steps below, or untouched for r = 0)
      if (s == 0) {
        stage(As, F + jc * N + jc, N, b, b);
        __syncthreads();
      }
      for (int e = t; e < 64 * 64; e += 256) {  // lower part, identity beyond b
        const int i = e >> 6, c = e & 63;
        if (i >= b || c >= b) As[i][c] = i == c ? cone<C>() : czero<C>();
        else if (c > i) As[i][c] = czero<C>();
      }
      C *Lb = Linv + (jc / 64) * 4096;
      const bool ok = ldlt_diag_phase1<C>(N, jc, b, F, err, smem_raw);
      if (ok)
        for (int e = t; e < 4 * 256; e += 256) {
          const int q = e >> 8, i = (e >> 4) & 15, c = e & 15;
          Lb[(16 * q + i) * 64 + 16 * q + c] = sm.Xd[q][i][c];
        }
      publish(diag_flag + s);
      // e of the panel's columns, 4^e about |D|: what balances W and L for the
      // int8 updates
      if (bal && ok && t < b) {
        int e;
        frexp(fmax(fabs((double)As[t][t].x), fabs((double)As[t][t].y)), &e);
        bal[jc + t] = (short)(e >> 1);
      }
      if (ok) ldlt_diag_phase2<C>(Lb, smem_raw);
      return;
    }
    // acc = -A_rs + sum_q W_rq L_sq^T
    {
      MidAcc<C, false> acc;
      acc.each([&](int i, int c, int e) {
        acc.set(e, (i < nr && c < b) ? cneg(__ldcg(F + (r0 + i) * N + jc + c)) : czero<C>());
      });
      for (int q = 0; q < s; q++) {
        if (!wait(row_flag + 4 * s + q)) return;
        stage(As, W + r0 * wstride + 64 * q, wstride, nr, 64);
        stage(Ls, F + jc * N + J + 64 * q, N, b, 64);
        __syncthreads();
        acc.mul(As, Ls);
        __syncthreads();
      }
      acc.each([&](int i, int c, int e) { As[i][c] = cneg(acc.get(e)); });
    }
    if (!wait(diag_flag + s)) return;
    stage(Ls, F + jc * N + jc, N, b, b);
#pragma unroll
    for (int m = 0; m < 4; m++) {
      const int e = t + 256 * m, q = e >> 8, i = (e >> 4) & 15, c = e & 15;
      sm.Xd[q][i][c] = __ldcg(Linv + (jc / 64) * 4096 + (16 * q + i) * 64 + 16 * q + c);
    }
    __syncthreads();
    if (t < b) dinv[t] = pivot_inverse(Ls[t][t]);
    mid_substitute(As + 8 * warp, Ls, sm.Xd, b);  // W_rs, 8 rows per warp
    __syncthreads();
    const bool below = rt < nsb;   // tiles of the panel's diagonal part keep L_rs for their own update
    const bool last = rt == s + 1;  // the factorisation of this tile comes next
#pragma unroll 4
    for (int m = 0; m < 16; m++) {
      const int e = t + 256 * m, i = e >> 6, c = e & 63;
      const C v = c < b ? As[i][c] : czero<C>();
      const C l = c < b ? cmul(v, dinv[c]) : czero<C>();
      if (i < nr && c < b) {
        W[(r0 + i) * wstride + 64 * s + c] = v;
        F[(r0 + i) * N + jc + c] = l;
      }
      if (below) Ls[i][c] = l;
    }
    if (!below) {
      __syncthreads();
      continue;
    }
    if (last) __syncthreads();  // published after the update, when the stores have drained
    else publish(row_flag + 4 * rt + s);
    // the own diagonal tile -= W_rs L_rs^T
    MidAcc<C, true> acc;
    C fd[sizeof(C) == 16 ? 10 : 16];  // the tile's own elements, by the accumulator's index
    acc.each([&](int i, int c, int e) {
      fd[e] = (i < nr && c <= i) ? __ldcg(F + (r0 + i) * N + r0 + c) : czero<C>();
    });
    acc.mul(As, Ls);
    if (last) publish(row_flag + 4 * rt + s);
    else __syncthreads();
    acc.each([&](int i, int c, int e) {
      if (i >= nr || c > i) return;
      const C d = csub(fd[e], acc.get(e));
      if (last) As[i][c] = d;
      else __stcg(F + (r0 + i) * N + r0 + c, d);
    });
    __syncthreads();
  }
}

template <class FC>
__global__ void k_scale_by_dinv(int64_t N, int64_t R, const FC *__restrict__ F, double2 *__restrict__ x) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N * R) return;
  int64_t n = i % N;
  x[i] = cdiv(x[i], to_d2(F[n * N + n]));
}

__global__ void k_scale_vec(int64_t N, int64_t R, const double2 *__restrict__ d, double2 *__restrict__ x) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N * R) return;
  x[i] = cmul(x[i], d[i % N]);
}

// Three-level right-looking LDL^T.  Block columns of NBW = 1024 are factored
// as 256-wide middle panels (one launch each).  After each middle panel the rest
// of the 1024-wide block column receives one K = 256 update, and after the block
// column the whole trailing matrix receives one K = 1024 update -- on the tensor
// cores (complex64: split operands, complex128: int8 residues).
//
// Lookahead (details at update_block_column / update_trailing): the next panel's
// latency-bound launch and the update before it run on the main stream while the rest of each update streams through the tensor cores on two side
// streams, always on columns disjoint from the main stream's.
constexpr int NBO = 256;
constexpr int NBW = 1024;

// W is free once a factorisation is done.  Until the next one it holds the
// 256-row block inverses of the few-column sweeps and, behind them, the products
// of prepare_block_inverses: two allocations less for a context's first solve.
size_t inverse_products_at(int64_t N) { return sizeof(double2) * N * 256; }
size_t inverse_bytes(int64_t N) {
  const size_t few = sizeof(double2) * ((N + 255) / 256) * 256 * 64, many = sizeof(float2) * ((N + 1023) / 1024) * 1024 * 256;
  return inverse_products_at(N) + std::max(few, many);
}

template <class C> void ldlt_factor(dmb_ctx *c, C *F) {
  c->f_version++;  // F changes from here on: packed copies are stale
  const int64_t N = c->n;
  raise_smem(c, k_ldlt_mid<C>, DiagSmem<C>::bytes);
  const int nblk = (int)((N + NB - 1) / NB);
  c->d_W.ensure(std::max(sizeof(C) * N * NBW * 2, inverse_bytes(N)));
  c->d_dinv.ensure(sizeof(C) * (size_t)nblk * NB * NB);  // Linv blocks
  // err word, then the tickets and flags of each middle panel
  const size_t flag_words = 4 + MID_WORDS * (size_t)((N + NBO - 1) / NBO);
  c->d_flags.ensure(std::max<size_t>(64, 4 * flag_words));
  if (!c->stream2 || !c->stream3) {
    // the panel chain (context stream) first, then the lookahead updates,
    // then auxiliary work (right-hand sides, int8 operand planes), which only
    // fills SMs the factorisation leaves idle
    int least = 0, greatest = 0;
    DMB_CUDA(cudaDeviceGetStreamPriorityRange(&least, &greatest));
    const int mid = greatest < least ? greatest + 1 : least;
    if (!c->stream2) DMB_CUDA(cudaStreamCreateWithPriority(&c->stream2, cudaStreamNonBlocking, mid));
    if (!c->stream3) DMB_CUDA(cudaStreamCreateWithPriority(&c->stream3, cudaStreamNonBlocking, mid));
  }
  for (auto &e : c->la_ev)
    if (!e) DMB_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  unsigned *err = c->d_flags.as<unsigned>();
  C *Linv = c->d_dinv.as<C>();
  unsigned *step_sync = err + 4;
  DMB_CUDA(cudaMemsetAsync(err, 0, 4 * flag_words, c->stream));
  const bool use_tc = std::is_same<C, float2>::value && dmb::tc_available(c);
  // complex128 updates on the int8 tensor cores: a first run through the schedule
  // only notes what each stream's largest update needs
  short *bal = nullptr;  // column exponents of the int8 updates; null: FP64 pipe
  bool planning = std::is_same<C, double2>::value && dmb::oz64_available(c, NBO);
  size_t need[3] = {0, 0, 0};
  // trailing update F[r][cc] -= W[r][woff..woff+K) L[cc][jcol..jcol+K) on
  // rows >= r0, columns [r0, c_hi); slot: the packed-operand buffers of the
  // issuing stream (0 main, 1 stream2, 2 stream3)
  auto update = [&](int64_t r0, int64_t c_hi, int64_t jcol, int K, const C *Wb, int woff, int slot) {
    const int64_t rest = N - r0;
    if (rest <= 0 || c_hi <= r0) return;
    if (planning) {
      need[slot] = std::max(need[slot], dmb::oz64_bytes(rest, c_hi - r0, K));
      return;
    }
    kt_begin(c);
    if (use_tc) {
      dmb::tc_ldlt_update_c64(c, N, r0, c_hi, jcol, K, (float2 *)F, (const float2 *)Wb, NBW, woff, slot);
    } else if constexpr (std::is_same<C, double2>::value) {
      const double2 *Wk = (const double2 *)Wb + r0 * NBW + woff, *Lk = (const double2 *)F + r0 * N + jcol;
      if (bal && dmb::oz64_available(c, K))
        dmb::oz64_lower_update(c, rest, c_hi - r0, K, Wk, NBW, Lk, N, bal + jcol, (double2 *)F + r0 * N + r0, N,
                               slot, err);
      else
        // the FP64-pipe GEMM (lower triangle)
        dmb::zgemm64_lower_update(c, rest, c_hi - r0, K, Wk, NBW, Lk, N, (double2 *)F + r0 * N + r0, N);
    } else {
      dim3 g(blocks_for(rest, 64), blocks_for(c_hi - r0, 64));
      DMB_LAUNCH(c, k_ldlt_update<C>, g, 256, 0, N, r0, c_hi, jcol, K, F, Wb, NBW, woff);
    }
    // algorithmic work: K complex MACs per updated lower-triangle entry
    const double cols = (double)(c_hi - r0), rows = (double)rest;
    kt_end(c, 8.0 * K * (cols * rows - cols * (cols - 1) / 2.0), 2);
  };
  // Lookahead.  Updates of one panel are split by columns: the next 256
  // columns on the main stream (the next panel needs them), the rest of the
  // current 1024-wide block column on stream2 and, for the trailing update at
  // the end of a block column, everything beyond the next block column on
  // stream3.  Concurrent updates always cover disjoint column ranges; before
  // an update of columns that a side stream may still be updating, the main
  // stream joins that stream (pend2 / pend3).  Each stream packs into its own
  // buffer slot, and W is double-buffered per block column, so a stream3
  // update may run through the whole next block column.
  bool pend2 = false, pend3 = false;
  auto join2 = [&] {
    if (pend2) DMB_CUDA(cudaStreamWaitEvent(c->stream, c->la_ev[1], 0));
    pend2 = false;
  };
  auto join3 = [&] {
    if (pend3) DMB_CUDA(cudaStreamWaitEvent(c->stream, c->la_ev[3], 0));
    pend3 = false;
  };
  // columns [lo, hi) updated on a side stream (1: stream2, 2: stream3) after
  // everything issued so far on the main stream
  auto side = [&](int which, int64_t lo, int64_t hi, int64_t jcol, int K, const C *Wb, int woff) {
    if (lo >= hi || lo >= N) return;
    if (planning) return update(lo, hi, jcol, K, Wb, woff, which);
    cudaStream_t s = which == 1 ? c->stream2 : c->stream3;
    cudaEvent_t start = c->la_ev[which == 1 ? 0 : 2], done = c->la_ev[which == 1 ? 1 : 3];
    DMB_CUDA(cudaEventRecord(start, c->stream));
    DMB_CUDA(cudaStreamWaitEvent(s, start, 0));
    {
      StreamSwap sw(c, s);
      update(lo, hi, jcol, K, Wb, woff, which);
    }
    DMB_CUDA(cudaEventRecord(done, s));
    (which == 1 ? pend2 : pend3) = true;
  };
  // after a 256-wide middle panel: the rest of its block column, and the
  // first 256 columns of the next block column (the next block column's first
  // panel): on stream3 behind the trailing update that also covers them, or,
  // after the block column's last panel, on the main stream once stream3 has
  // joined.  The trailing update at the block column's end then leaves those
  // 256 columns out, so no K = 1,024 update sits on the chain.
  auto update_block_column = [&](int64_t r0, int64_t c_hi, int64_t jcol, int K, const C *Wb, int woff) {
    join2();
    const int64_t cmid = std::min<int64_t>(c_hi, r0 + NBO);
    update(r0, cmid, jcol, K, Wb, woff, 0);
    side(1, cmid, c_hi, jcol, K, Wb, woff);
    const int64_t n0 = c_hi, n1 = std::min<int64_t>(N, c_hi + NBO);
    if (n0 < n1) {
      if (r0 >= c_hi) {  // the block column's last panel
        join3();
        update(n0, n1, jcol, K, Wb, woff, 0);
      } else {
        side(2, n0, n1, jcol, K, Wb, woff);
      }
    }
  };
  // after a block column: the trailing matrix beyond the next block column's
  // first panel
  auto update_trailing = [&](int64_t r0, int64_t jcol, int K, const C *Wb) {
    join2();
    join3();
    const int64_t c1 = std::min<int64_t>(N, r0 + NBO), c2 = std::min<int64_t>(N, r0 + NBW);
    side(1, c1, c2, jcol, K, Wb, 0);
    side(2, c2, N, jcol, K, Wb, 0);
  };
  auto schedule = [&] {
    int64_t bc = 0;
    for (int64_t J2 = 0; J2 < N; J2 += NBW, bc++) {
      C *Wb = c->d_W.as<C>() + (bc & 1) * N * NBW;
      const int64_t J2E = std::min<int64_t>(N, J2 + NBW);
      for (int64_t J = J2; J < J2E; J += NBO) {
        const int64_t JE = std::min<int64_t>(J2E, J + NBO);
        if (!planning)
          DMB_LAUNCH(c, k_ldlt_mid<C>, blocks_for(N - J, NB), 256, DiagSmem<C>::bytes, N, J, (int)(JE - J), F, Linv,
                     Wb + (J - J2), NBW, bal, step_sync + MID_WORDS * (J / NBO), err, c->spin_limit);
        update_block_column(JE, J2E, J, (int)(JE - J), Wb, (int)(J - J2));
      }
      update_trailing(J2E, J2, (int)(J2E - J2), Wb);
    }
  };
  if (planning) {
    schedule();
    planning = false;
    if (need[0] > 0 && dmb::oz64_reserve(c, N, need)) bal = c->oz64.buf.as<short>();
  }
  schedule();
  join2();
  join3();
  unsigned h_err = 0;
  DMB_CUDA(cudaMemcpyAsync(&h_err, err, 4, cudaMemcpyDeviceToHost, c->stream));
  DMB_CUDA(cudaStreamSynchronize(c->stream));
  DMB_REQUIRE(!(h_err & 4u), DMB_ERR_TIMEOUT, "factorisation: a panel-step wait expired");
  DMB_REQUIRE(!(h_err & 8u), DMB_ERR_TIMEOUT, "int8 tensor-core update: a pipeline wait expired");
  DMB_REQUIRE(h_err == 0, DMB_ERR_BREAKDOWN, "near-field factorisation broke down: zero or non-finite pivot");
  if (use_tc)
    DMB_REQUIRE(dmb::tc_error_word(c) == 0, DMB_ERR_TIMEOUT, "tensor-core update: a pipeline wait expired");
}

// ---------------------------------------------------------------------------
// Batched triangular solves for many right-hand sides (X column-major N x R).
// The factor is walked in 256-row panels: the in-panel part (four 64-blocks
// with their stored Linv) runs in k_trsm_panel, where one CTA owns TP_COLS
// right-hand sides; the rest of the rows receive one GEMM-shaped update per
// panel (tensor cores for the complex64 factor, SIMT otherwise).  F is read
// once per sweep instead of once per right-hand side.
// ---------------------------------------------------------------------------
constexpr int TP = 256;      // panel rows
constexpr int TP_COLS = 8;   // right-hand sides per CTA

// T[i][j] <- G(i, j) for i, j < 64 (zero outside bi x bj); TR reads G(j, i)
template <class FC, bool TR>
__device__ __forceinline__ void stage_tile(FC (*T)[65], const FC *__restrict__ G, int64_t ld, int bi, int bj) {
  for (int e = threadIdx.x; e < 64 * 64; e += 256) {
    const int a = e >> 6, b = e & 63;  // consecutive threads: consecutive b
    if (TR) {
      // element (i = b, j = a) = G[a * ld + b]
      T[b][a] = (b < bi && a < bj) ? G[(int64_t)a * ld + b] : FC{};
    } else {
      T[a][b] = (a < bi && b < bj) ? G[(int64_t)a * ld + b] : FC{};
    }
  }
}

template <class FC, bool BWD>
__global__ void __launch_bounds__(256) k_trsm_panel(int64_t N, int64_t R, int64_t p0, int width,
                                                    const FC *__restrict__ F, const FC *__restrict__ Linv,
                                                    double2 *__restrict__ X) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  FC(*T)[65] = reinterpret_cast<FC(*)[65]>(smem_raw);
  double2(*xs)[TP_COLS + 1] = reinterpret_cast<double2(*)[TP_COLS + 1]>(smem_raw + sizeof(FC) * 64 * 65);
  const int64_t r0 = (int64_t)blockIdx.x * TP_COLS;
  for (int e = threadIdx.x; e < width * TP_COLS; e += 256) {
    const int q = e / width, i = e % width;
    xs[i][q] = (r0 + q < R) ? X[(r0 + q) * N + p0 + i] : make_double2(0, 0);
  }
  const int nb = (width + 63) / 64;
  const int i = threadIdx.x & 63, qh = threadIdx.x >> 6;  // rows i, columns qh and qh + 4
  for (int s = 0; s < nb; s++) {
    const int b = BWD ? nb - 1 - s : s;
    const int bs = min(64, width - 64 * b);
    const int64_t t = (p0 >> 6) + b;  // global 64-block index
    __syncthreads();
    // BWD: x_b = Linv_b^T y_b, FWD: y_b = Linv_b x_b
    stage_tile<FC, BWD>(T, Linv + t * 4096, 64, bs, bs);
    __syncthreads();
    double2 acc0 = make_double2(0, 0), acc1 = make_double2(0, 0);
    if (i < bs) {
      for (int j = 0; j < bs; j++) {
        const double2 l = to_d2(T[i][j]);
        cfma(acc0, l, xs[64 * b + j][qh]);
        cfma(acc1, l, xs[64 * b + j][qh + 4]);
      }
    }
    __syncthreads();
    if (i < bs) {
      xs[64 * b + i][qh] = acc0;
      xs[64 * b + i][qh + 4] = acc1;
    }
    // the other blocks of the panel that depend on block b
    for (int s2 = s + 1; s2 < nb; s2++) {
      const int b2 = BWD ? nb - 1 - s2 : s2;
      const int bs2 = min(64, width - 64 * b2);
      __syncthreads();
      if (BWD)  // x_{b2} -= L[b, b2]^T x_b : T[i][j] = L[p0 + 64 b + j][p0 + 64 b2 + i]
        stage_tile<FC, true>(T, F + (p0 + 64 * b) * N + p0 + 64 * b2, N, bs2, bs);
      else      // y_{b2} -= L[b2, b] y_b  : T[i][j] = L[p0 + 64 b2 + i][p0 + 64 b + j]
        stage_tile<FC, false>(T, F + (p0 + 64 * b2) * N + p0 + 64 * b, N, bs2, bs);
      __syncthreads();
      if (i < bs2) {
        double2 u0 = make_double2(0, 0), u1 = make_double2(0, 0);
        for (int j = 0; j < bs; j++) {
          const double2 l = to_d2(T[i][j]);
          cfma(u0, l, xs[64 * b + j][qh]);
          cfma(u1, l, xs[64 * b + j][qh + 4]);
        }
        xs[64 * b2 + i][qh] = csub(xs[64 * b2 + i][qh], u0);
        xs[64 * b2 + i][qh + 4] = csub(xs[64 * b2 + i][qh + 4], u1);
      }
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < width * TP_COLS; e += 256) {
    const int q = e / width, ii = e % width;
    if (r0 + q < R) X[(r0 + q) * N + p0 + ii] = xs[ii][q];
  }
}

// SIMT panel update  Y[m, r] -= sum_k A(m, k) B[k, r]  (FP64 accumulation),
// A(m, k) = A[m lda + k] or, TR, A[k lda + m]; B, Y column-major.  64 x 64
// output tiles, K in chunks of 16.
template <class FC, bool TR>
__global__ void __launch_bounds__(256) k_gemm_sub(int64_t M, int64_t R, int K, const FC *__restrict__ A, int64_t lda,
                                                  const double2 *__restrict__ B, int64_t ldb, double2 *__restrict__ Y,
                                                  int64_t ldy) {
  __shared__ double2 As[16][65];
  __shared__ double2 Bs[16][65];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int64_t m0 = (int64_t)blockIdx.x * 64, r0 = (int64_t)blockIdx.y * 64;
  double2 acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int b = 0; b < 4; b++) acc[a][b] = make_double2(0, 0);
  for (int k0 = 0; k0 < K; k0 += 16) {
    for (int e = threadIdx.x; e < 16 * 64; e += 256) {
      int kk, mm;
      if (TR) { mm = e & 63; kk = e >> 6; } else { kk = e & 15; mm = e >> 4; }
      const int64_t m = m0 + mm;
      const int kx = k0 + kk;
      As[kk][mm] = (m < M && kx < K) ? to_d2(TR ? A[(int64_t)kx * lda + m] : A[m * lda + kx]) : make_double2(0, 0);
      const int kb = e & 15, rb = e >> 4;
      const int64_t r = r0 + rb;
      Bs[kb][rb] = (r < R && k0 + kb < K) ? B[r * ldb + k0 + kb] : make_double2(0, 0);
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < 16; kk++) {
      double2 a[4], b[4];
#pragma unroll
      for (int u = 0; u < 4; u++) a[u] = As[kk][ty + 16 * u];
#pragma unroll
      for (int v = 0; v < 4; v++) b[v] = Bs[kk][tx + 16 * v];
#pragma unroll
      for (int u = 0; u < 4; u++)
#pragma unroll
        for (int v = 0; v < 4; v++) cfma(acc[u][v], a[u], b[v]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int u = 0; u < 4; u++)
#pragma unroll
    for (int v = 0; v < 4; v++) {
      const int64_t m = m0 + ty + 16 * u, r = r0 + tx + 16 * v;
      if (m < M && r < R) Y[r * ldy + m] = csub(Y[r * ldy + m], acc[u][v]);
    }
}

template <class C> constexpr size_t trsm_panel_smem() {
  return sizeof(C) * 64 * 65 + sizeof(double2) * TP * (TP_COLS + 1);
}
template <class C> void trsm_panel_attrs(dmb_ctx *c) {
  raise_smem(c, k_trsm_panel<C, false>, trsm_panel_smem<C>());
  raise_smem(c, k_trsm_panel<C, true>, trsm_panel_smem<C>());
}

// X[r_lo : r_hi] -= L[r_lo : r_hi, k_lo : k_lo + w] X[k_lo : k_lo + w]   (forward)
// X[r_lo : r_hi] -= L[k_lo : k_lo + w, r_lo : r_hi]^T X[k_lo : k_lo + w] (backward)
template <class C> void trsm_update(dmb_ctx *c, const C *F, int64_t N, int64_t r_lo, int64_t r_hi, int64_t k_lo,
                                    int w, bool bwd, double2 *X, int64_t R) {
  const int64_t M = r_hi - r_lo;
  if (M <= 0) return;
  if (std::is_same<C, float2>::value && R >= c->tc_min_rhs && dmb::tc_available(c)) {
    dmb::tc_trsm_update(c, (const float2 *)F, N, r_lo, r_hi, k_lo, w, bwd, X, R);
    return;
  }
  if constexpr (std::is_same<C, double2>::value) {
    if (M >= 128 && R >= 16) {  // complex128 factor: the FP64-pipe GEMM
      if (bwd)
        dmb::zgemm64_sub(c, true, M, R, w, F + k_lo * N + r_lo, N, X + k_lo, N, X + r_lo, N);
      else
        dmb::zgemm64_sub(c, false, M, R, w, F + r_lo * N + k_lo, N, X + k_lo, N, X + r_lo, N);
      return;
    }
  }
  dim3 g(blocks_for(M, 64), blocks_for(R, 64));
  if (bwd)
    DMB_LAUNCH(c, (k_gemm_sub<C, true>), g, 256, 0, M, R, w, F + k_lo * N + r_lo, N, X + k_lo, N, X + r_lo, N);
  else
    DMB_LAUNCH(c, (k_gemm_sub<C, false>), g, 256, 0, M, R, w, F + r_lo * N + k_lo, N, X + k_lo, N, X + r_lo, N);
}

// Two levels: 1024-row outer panels whose rows below (forward) / above
// (backward) receive one K = 1024 update, and inside each outer panel
// 256-row panels solved by k_trsm_panel with K = 256 updates restricted to
// the outer panel.
constexpr int TP_OUTER = 1024;

// forward solve restricted to rows [o0, o1): L[o0:o1, o0:o1] y = x
template <class C> void forward_block(dmb_ctx *c, const C *F, int64_t o0, int64_t o1, double2 *X, int64_t R) {
  const int64_t N = c->n;
  const size_t sm = trsm_panel_smem<C>();
  for (int64_t p0 = o0; p0 < o1; p0 += TP) {
    const int w = (int)std::min<int64_t>(TP, o1 - p0);
    DMB_LAUNCH(c, (k_trsm_panel<C, false>), blocks_for(R, TP_COLS), 256, sm, N, R, p0, w, F, c->d_dinv.as<C>(), X);
    trsm_update<C>(c, F, N, p0 + w, o1, p0, w, false, X, R);
  }
}

// Inverses of the OB-row diagonal blocks of the unit lower factor (OB = 1024
// for the tensor-core sweeps, 256 for the few-column ones) by recursive
// doubling from the 64 x 64 block inverses of the factorisation: for
// consecutive s-blocks A, B inside one outer block,
//   [A 0; C B]^-1 = [A^-1 0; -B^-1 C A^-1  B^-1],
// s = 64, 128, .. OB / 2, all pairs of a level in one launch per product.
// X (column-major, leading dimension N; outer block o occupies rows o0..o1 and
// block-local columns 0..o1-o0) receives the inverses.

// X <- the 64-block inverses on the diagonal of every outer block, 0 elsewhere
template <int OB, class FC>
__global__ void k_inv_init(int64_t N, const FC *__restrict__ Linv, double2 *__restrict__ X) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N * OB) return;
  const int64_t col = i / N, r = i % N;  // consecutive threads: consecutive rows
  const int64_t o0 = r - r % OB;
  double2 v = make_double2(0.0, 0.0);
  if (o0 + col < N && (o0 + col) / NB == r / NB) {
    v = to_d2(Linv[(r / NB) * NB * NB + (r % NB) * NB + (o0 + col) % NB]);
  }
  X[col * N + r] = v;
}

template <class TC> __device__ __forceinline__ TC inv_conv(double2 v);
template <> __device__ __forceinline__ float2 inv_conv<float2>(double2 v) { return make_float2((float)v.x, (float)v.y); }
template <> __device__ __forceinline__ double2 inv_conv<double2>(double2 v) { return v; }

// one product of a doubling level; pair slot y of outer block y / ppo covers
// A = [i0, i0 + s), B = [i0 + s, i0 + s + sb), i0 = o0 + 2 s (y % ppo)
//   STEP 1: T = F[B, A] (strict lower part of L) x A^-1     (sb x s)
//   STEP 2: X[B, A] = -B^-1 x T                             (sb x s)
// 64 x 64 output tiles (grid.x), FP32 SIMT with 16-deep shared stages
// TC: the arithmetic of the products (float2 for the tensor-core sweeps'
// inverses, double2 for the one-RHS sweeps')
template <int STEP, int OB, class FC, class TC>
__global__ void __launch_bounds__(256) k_inv_level(int64_t N, int s, const FC *__restrict__ F,
                                                   double2 *__restrict__ X, TC *__restrict__ T) {
  __shared__ TC As[16][65];
  __shared__ TC Bs[16][65];
  const int ppo = OB / (2 * s);
  const int64_t o0 = (int64_t)(blockIdx.y / ppo) * OB;
  const int64_t o1 = min(N, o0 + OB);
  const int64_t i0 = o0 + 2 * (int64_t)s * (blockIdx.y % ppo);
  const int64_t a0 = i0, b0 = i0 + s;
  if (b0 >= o1) return;  // no B block in this slot
  const int sb = (int)min((int64_t)s, o1 - b0);
  const int nt = (s + 63) / 64;
  const int ti = blockIdx.x / nt, tj = blockIdx.x % nt;
  if (64 * ti >= sb) return;
  TC *Tp = T + (int64_t)blockIdx.y * s * s;  // column-major sb x s, leading dimension s
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  TC acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = czero<TC>();
  // STEP 1: k runs over A's columns from the tile's first column (A^-1 is
  // lower); STEP 2: over B's columns up to the tile's last row (B^-1 is lower)
  const int k_lo = STEP == 1 ? 64 * tj : 0;
  const int k_hi = STEP == 1 ? s : min(sb, 64 * ti + 64);
  for (int k0 = k_lo; k0 < k_hi; k0 += 16) {
    for (int e = threadIdx.x; e < 16 * 64; e += 256) {
      if (STEP == 1) {
        const int kk = e & 15, rr = e >> 4;  // k fastest: F rows and X columns are k-contiguous
        const int k = k0 + kk, i = 64 * ti + rr, j = 64 * tj + rr;
        const FC f = (k < k_hi && i < sb) ? F[(b0 + i) * N + a0 + k] : czero<FC>();
        As[kk][rr] = inv_conv<TC>(to_d2(f));
        const double2 x = (k < k_hi) ? X[(a0 - o0 + j) * N + a0 + k] : make_double2(0.0, 0.0);
        Bs[kk][rr] = inv_conv<TC>(x);
      } else {
        const int rr = e & 63, kk = e >> 6;  // rows fastest for B^-1 (column-major)
        const int k = k0 + kk, i = 64 * ti + rr;
        const double2 x = (k < k_hi && i < sb) ? X[(b0 - o0 + k) * N + b0 + i] : make_double2(0.0, 0.0);
        As[kk][rr] = inv_conv<TC>(x);
        const int kk2 = e & 15, cc = e >> 4, k2 = k0 + kk2, j = 64 * tj + cc;
        Bs[kk2][cc] = (k2 < k_hi && j < s) ? Tp[(int64_t)j * s + k2] : czero<TC>();
      }
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < 16; kk++) {
      TC a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; i++) a[i] = As[kk][ty + 16 * i];
#pragma unroll
      for (int j = 0; j < 4; j++) b[j] = Bs[kk][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) cfma(acc[i][j], a[i], b[j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int r = 64 * ti + ty + 16 * i, cidx = 64 * tj + tx + 16 * j;
      if (r >= sb || cidx >= s) continue;
      if (STEP == 1)
        Tp[(int64_t)cidx * s + r] = acc[i][j];
      else
        X[(a0 - o0 + cidx) * N + b0 + r] = make_double2(-(double)acc[i][j].x, -(double)acc[i][j].y);
    }
}

// The block inverses of L (once per factorisation): 1024-row ones by FP32
// products into d_trsm_id for the tensor-core sweeps (which round them to TF32
// anyway), 256-row ones by FP64 products into W for the few-column sweeps (as
// accurate as substitution with the stored 64-block inverses).
template <int OB, class FC, class TC>
void prepare_block_inverses(dmb_ctx *c, const FC *F, double2 *Xid, uint64_t &ver) {
  if (ver == c->f_version) return;
  const int64_t N = c->n;
  const int64_t nout = (N + OB - 1) / OB;
  // the products T: (pair slots) x s x s <= nout x OB x OB / 4
  TC *T = reinterpret_cast<TC *>(c->d_W.as<char>() + inverse_products_at(N));
  DMB_LAUNCH(c, (k_inv_init<OB, FC>), blocks_for(N * OB, 256), 256, 0, N, c->d_dinv.as<FC>(), Xid);
  for (int s = NB; s < OB && s < N; s *= 2) {
    const int nt = (s + 63) / 64;
    dim3 g((unsigned)(nt * nt), (unsigned)(nout * (OB / (2 * s))));
    DMB_LAUNCH(c, (k_inv_level<1, OB, FC, TC>), g, 256, 0, N, s, F, Xid, T);
    DMB_LAUNCH(c, (k_inv_level<2, OB, FC, TC>), g, 256, 0, N, s, F, Xid, T);
  }
  ver = c->f_version;
}

// Pack the complex64 factor for the tensor-core sweeps (once per
// factorisation): L'' and (L^T)'', and the 1024-row block inverses.
void prepare_packed_factor(dmb_ctx *c, const float2 *F) {
  if (c->f_packed == c->f_version) return;
  const int64_t N = c->n;
  trsm_panel_attrs<float2>(c);
  dmb::tc_trsm_pack_factor(c, F, N);
  c->d_trsm_id.ensure(sizeof(double2) * N * TP_OUTER);
  double2 *Xid = c->d_trsm_id.as<double2>();
  prepare_block_inverses<TP_OUTER, float2, float2>(c, F, Xid, c->f_inv);
  const int64_t nout = (N + TP_OUTER - 1) / TP_OUTER;
  for (int64_t o = 0; o < nout; o++) {
    const int64_t o0 = o * TP_OUTER, o1 = std::min<int64_t>(N, o0 + TP_OUTER);
    dmb::tc_trsm_pack_diag(c, o, Xid + o0, N, (int)(o1 - o0));
  }
  c->f_packed = c->f_version;
}

// ---------------------------------------------------------------------------
// Triangular sweeps for one to seven right-hand sides (one per grid.y), L and
// its transpose, by data flow over 256-row blocks:
//   forward,  o = 0..last: a_o = b_o - L[o, <o] y,       y_o = X_o a_o
//   backward, o = last..0: a_o = y_o / D - L[>o, o]^T x, x_o = X_o^T a_o
// with X_o the inverse of L's diagonal block.  A CTA owns 16 rows (forward) or
// columns (backward) of a block: it streams its part of L block by block as the
// blocks of y (x) appear, publishes its 16 values of a_o, and, once the part of
// a_o that its rows of X_o need is there, its 16 values of X_o a_o.  The values are their own flags: the
// buffers are filled with a bit pattern that no published value has (SV_EMPTY),
// and a thread that needs a value reads it until it is there.  The next block's
// part of L is loaded ahead of that, the part of X_o at the start, so a block
// costs two trips through L2 and two short sums; the stream of L runs beside
// that chain over all SMs.  CTAs take their slices in ticket order (forward
// sweep downwards, backward upwards) and wait only on earlier tickets -- of their
// own block too, X_o being triangular -- so a sweep goes on however few of its
// CTAs are resident; every wait is bounded (error bit 4).  All sums in a fixed
// order.  Bound by the chain up to N = 10,000 and by the read of L above.
// Measured, both sweeps: complex128 415 us at N = 10,680 (912 MB of L each), 56 us
// at 1,825; complex64 177 us at 4,693.  With counters as flags (two
// barriers, a fence and an atomic a hand-over): 640, 95 and 260 us.
// ---------------------------------------------------------------------------
constexpr int SV = 256;  // rows per block
constexpr int SW = 16;   // rows per CTA
constexpr int SV_LD = SV + 1;
constexpr unsigned long long SV_EMPTY = ~0ull;  // a NaN; published NaNs are made to differ from it

__device__ __forceinline__ void sv_publish(double2 *p, double2 v) {
  unsigned long long x = __double_as_longlong(v.x), y = __double_as_longlong(v.y);
  if (x == SV_EMPTY) x = 0x7ff8000000000000ull;
  if (y == SV_EMPTY) y = 0x7ff8000000000000ull;
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(x), "l"(y) : "memory");
}

// The values lo to n - 1 at p into v[0..255] (zero elsewhere), a thread each, as
// they are published; for the whole CTA, false on expiry or another CTA's.  v is
// read after, and written before, the next barrier.
__device__ __forceinline__ bool sv_gather(const double2 *p, int lo, int n, double2 *v, int64_t ahead, unsigned *err,
                                          long long limit) {
  const int t = threadIdx.x;
  bool ok = true;
  unsigned long long x = 0, y = 0;
  if (t >= lo && t < n) {
    for (long long it = 0;;) {
      asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "l"(p + t) : "memory");
      if (x != SV_EMPTY && y != SV_EMPTY) break;
      if (++it > limit) {
        atomicOr(err, 4u);
        ok = false;
        break;
      }
      if ((it & 15) == 0 && (*((volatile unsigned *)err) & 4u)) {
        ok = false;
        break;
      }
      // blocks ahead of the chain leave L2 to it
      if (ahead > 1) __nanosleep(ahead > 3 ? 500 : 100);
      else if (it > 64) __nanosleep(20);
    }
  }
  v[t] = make_double2(__longlong_as_double((long long)x), __longlong_as_double((long long)y));
  return __syncthreads_and(ok);
}

// sums of a warp's two rows m (entries lane + 32 j) times v
__device__ __forceinline__ void rows2_fma(const double2 *m, const double2 *v, int lane, double2 &s0, double2 &s1) {
#pragma unroll
  for (int j = 0; j < 8; j++) {
    const double2 y = v[lane + 32 * j];
    cfma(s0, m[lane + 32 * j], y);
    cfma(s1, m[SV_LD + lane + 32 * j], y);
  }
}

__global__ void k_sweep_clear(int64_t n, ulonglong2 *buf, int ntickets, unsigned *tickets) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e < n) buf[e] = make_ulonglong2(SV_EMPTY, SV_EMPTY);
  if (e < ntickets) tickets[e] = 0u;
}

struct SweepSmem {
  double2 X[SW][SV_LD];  // the CTA's rows of the block inverse (its transpose)
  double2 v[2][SV];      // blocks in turn
  double2 red[8][SW];
};

template <class FC>
__global__ void __launch_bounds__(256, 2) k_sweep_fwd(int64_t N, const FC *__restrict__ F,
                                                      const double2 *__restrict__ X, const double2 *__restrict__ b,
                                                      double2 *abuf, double2 *y, unsigned *tickets, unsigned *err,
                                                      long long limit) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SweepSmem &sm = *reinterpret_cast<SweepSmem *>(smem_raw);
  constexpr bool AHEAD = sizeof(FC) == 8;  // room in registers for two blocks of L
  __shared__ int s_t;
  const int rhs = blockIdx.y, t = threadIdx.x, warp = t >> 5, lane = t & 31;
  b += rhs * N;
  abuf += rhs * N;
  y += rhs * N;
  if (t == 0) s_t = (int)atomicAdd(tickets + rhs, 1u);
  __syncthreads();
  const int64_t r0 = (int64_t)s_t * SW, o = r0 / SV, o0 = o * SV;
  const int nr = (int)min((int64_t)SW, N - r0);
  for (int e = t; e < SW * SV; e += 256) {  // the inverse is kept transposed
    const int c = e & 15, k = e >> 4;
    sm.X[c][k] = (c < nr && k <= r0 - o0 + c) ? X[(int64_t)k * N + r0 + c] : make_double2(0.0, 0.0);
  }
  const int64_t ra = r0 + 2 * warp;  // this warp's rows ra, ra + 1
  const double2 br = lane < 2 && 2 * warp + lane < nr ? b[ra + lane] : make_double2(0.0, 0.0);
  double2 s0 = make_double2(0.0, 0.0), s1 = s0;
  auto load = [&](FC(&m)[16], int64_t p) {
    if (p >= o) return;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      m[j] = ra < N ? F[ra * N + p * SV + lane + 32 * j] : czero<FC>();
      m[8 + j] = ra + 1 < N ? F[(ra + 1) * N + p * SV + lane + 32 * j] : czero<FC>();
    }
  };
  // block p of L, already loaded (complex64: the next one's loads on their way)
  auto step = [&](FC(&m)[16], FC(&next)[16], int64_t p) {
    if (AHEAD) load(next, p + 1);
    else load(m, p);
    if (!sv_gather(y + p * SV, 0, SV, sm.v[p & 1], o - p, err, limit)) return false;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const double2 yv = sm.v[p & 1][lane + 32 * j];
      cfma(s0, to_d2(m[j]), yv);
      cfma(s1, to_d2(m[8 + j]), yv);
    }
    return true;
  };
  FC ma[16], mb[16];
  if (AHEAD) load(ma, 0);
  for (int64_t p = 0; p < o; p += 2) {
    if (!step(ma, mb, p)) return;
    if (p + 1 < o && !step(mb, ma, p + 1)) return;
  }
  s0 = warp_sum2(s0);
  s1 = warp_sum2(s1);
  if (lane < 2 && 2 * warp + lane < nr) sv_publish(abuf + ra + lane, csub(br, lane == 0 ? s0 : s1));
  // X_o is lower triangular: the rows up to this CTA's, of earlier tickets
  if (!sv_gather(abuf + o0, 0, (int)(r0 - o0) + nr, sm.v[o & 1], 0, err, limit)) return;
  s0 = s1 = make_double2(0.0, 0.0);
  rows2_fma(sm.X[2 * warp], sm.v[o & 1], lane, s0, s1);
  s0 = warp_sum2(s0);
  s1 = warp_sum2(s1);
  if (lane < 2 && 2 * warp + lane < nr) sv_publish(y + ra + lane, lane == 0 ? s0 : s1);
}

template <class FC>
__global__ void __launch_bounds__(256, 2) k_sweep_bwd(int64_t N, const FC *__restrict__ F,
                                                      const double2 *__restrict__ X, const double2 *__restrict__ y,
                                                      double2 *abuf, double2 *xbuf, double2 *x, unsigned *tickets,
                                                      unsigned *err, long long limit) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SweepSmem &sm = *reinterpret_cast<SweepSmem *>(smem_raw);
  constexpr bool AHEAD = sizeof(FC) == 8;  // room in registers for two blocks of L
  __shared__ int s_t;
  const int rhs = blockIdx.y, t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int64_t nblk = (N + SV - 1) / SV;
  y += rhs * N;
  abuf += rhs * N;
  xbuf += rhs * N;
  x += rhs * N;
  if (t == 0) s_t = (int)atomicAdd(tickets + rhs, 1u);
  __syncthreads();
  const int64_t r0 = ((N + SW - 1) / SW - 1 - s_t) * SW, o = r0 / SV, o0 = o * SV;
  const int nr = (int)min((int64_t)SW, N - r0), w = (int)min((int64_t)SV, N - o0);
  for (int e = t; e < SW * SV; e += 256) {
    const int c = e >> 8, k = e & 255;
    sm.X[c][k] = (c < nr && k >= r0 - o0 + c && k < w) ? X[(r0 - o0 + c) * N + o0 + k] : make_double2(0.0, 0.0);
  }
  double2 yd = make_double2(0.0, 0.0);
  if (t < nr) yd = cdiv(y[r0 + t], to_d2(F[(r0 + t) * N + r0 + t]));
  const int c = t & 15, g = t >> 4;  // column r0 + c, rows g + 16 j of a block
  double2 v = make_double2(0.0, 0.0);
  auto load = [&](FC(&m)[16], int64_t p) {
    if (p <= o) return;
    const int n = (int)min((int64_t)SV, N - p * SV);
#pragma unroll
    for (int j = 0; j < 16; j++)
      m[j] = (g + 16 * j < n && c < nr) ? F[(p * SV + g + 16 * j) * N + r0 + c] : czero<FC>();
  };
  auto step = [&](FC(&m)[16], FC(&next)[16], int64_t p) {
    if (AHEAD) load(next, p - 1);
    else load(m, p);
    if (!sv_gather(xbuf + p * SV, 0, (int)min((int64_t)SV, N - p * SV), sm.v[p & 1], p - o, err, limit)) return false;
#pragma unroll
    for (int j = 0; j < 16; j++) cfma(v, to_d2(m[j]), sm.v[p & 1][g + 16 * j]);
    return true;
  };
  FC ma[16], mb[16];
  if (AHEAD) load(ma, nblk - 1);
  for (int64_t p = nblk - 1; p > o; p -= 2) {
    if (!step(ma, mb, p)) return;
    if (p - 1 > o && !step(mb, ma, p - 1)) return;
  }
  // sum of the 16 row groups
  v.x += __shfl_xor_sync(0xffffffffu, v.x, 16);
  v.y += __shfl_xor_sync(0xffffffffu, v.y, 16);
  if (lane < 16) sm.red[warp][lane] = v;
  __syncthreads();
  if (t < nr) {
    double2 s = make_double2(0.0, 0.0);
#pragma unroll
    for (int q = 0; q < 8; q++) s = cadd(s, sm.red[q][t]);
    sv_publish(abuf + r0 + t, csub(yd, s));
  }
  // X_o^T is upper triangular: the rows from this CTA's on, of earlier tickets
  if (!sv_gather(abuf + o0, (int)(r0 - o0), w, sm.v[o & 1], 0, err, limit)) return;
  double2 s0 = make_double2(0.0, 0.0), s1 = s0;
  rows2_fma(sm.X[2 * warp], sm.v[o & 1], lane, s0, s1);
  s0 = warp_sum2(s0);
  s1 = warp_sum2(s1);
  if (lane < 2 && 2 * warp + lane < nr) {
    const double2 r = lane == 0 ? s0 : s1;
    sv_publish(xbuf + r0 + 2 * warp + lane, r);
    x[r0 + 2 * warp + lane] = r;
  }
}

template <class C> void ldlt_solve(dmb_ctx *c, const C *F, double2 *x, int64_t R) {
  const int64_t N = c->n;
  double2 *X = c->d_W.as<double2>();
  prepare_block_inverses<SV, C, double2>(c, F, X, c->f_inv64);
  raise_smem(c, k_sweep_fwd<C>, sizeof(SweepSmem));
  raise_smem(c, k_sweep_bwd<C>, sizeof(SweepSmem));
  // a and y of the forward sweep, a and x of the backward one, all empty
  c->d_sv_acc.ensure(sizeof(double2) * 4 * N * R);
  double2 *buf = c->d_sv_acc.as<double2>();
  // the error word, then a ticket counter per column and sweep (at most 14; the
  // factorisation made room).  The error word stays: a solve's later sweeps must
  // not hide that an earlier one gave up (clear_err_word at the solve's start)
  unsigned *err = c->d_flags.as<unsigned>(), *tickets = err + 1;
  DMB_LAUNCH(c, k_sweep_clear, blocks_for(4 * N * R, 256), 256, 0, 4 * N * R, reinterpret_cast<ulonglong2 *>(buf),
             (int)(2 * R), tickets);
  const dim3 g((unsigned)((N + SW - 1) / SW), (unsigned)R);
  DMB_LAUNCH(c, k_sweep_fwd<C>, g, 256, sizeof(SweepSmem), N, F, X, x, buf, buf + N * R, tickets, err, c->spin_limit);
  DMB_LAUNCH(c, k_sweep_bwd<C>, g, 256, sizeof(SweepSmem), N, F, X, buf + N * R, buf + 2 * N * R, buf + 3 * N * R, x,
             tickets + R, err, c->spin_limit);
}

template <class C> void ldlt_solve_batched(dmb_ctx *c, const C *F, double2 *X, int64_t R) {
  const int64_t N = c->n;
  const C *Linv = c->d_dinv.as<C>();
  trsm_panel_attrs<C>(c);
  if (std::is_same<C, float2>::value && R >= c->tc_min_rhs && dmb::tc_available(c)) {
    // tensor cores: every step is a GEMM on operands packed once per factor
    prepare_packed_factor(c, (const float2 *)F);
    dmb::tc_trsm_sweep(c, N, X, R, false);
    DMB_LAUNCH(c, k_scale_by_dinv<C>, blocks_for(N * R, 256), 256, 0, N, R, F, X);
    dmb::tc_trsm_sweep(c, N, X, R, true);
    return;
  }
  const size_t sm = trsm_panel_smem<C>();
  const unsigned gcols = blocks_for(R, TP_COLS);
  const int64_t nout = (N + TP_OUTER - 1) / TP_OUTER;
  for (int64_t o = 0; o < nout; o++) {
    const int64_t o0 = o * TP_OUTER, o1 = std::min<int64_t>(N, o0 + TP_OUTER);
    forward_block<C>(c, F, o0, o1, X, R);
    trsm_update<C>(c, F, N, o1, N, o0, (int)(o1 - o0), false, X, R);
  }
  DMB_LAUNCH(c, k_scale_by_dinv<C>, blocks_for(N * R, 256), 256, 0, N, R, F, X);
  for (int64_t o = nout - 1; o >= 0; o--) {
    const int64_t o0 = o * TP_OUTER, o1 = std::min<int64_t>(N, o0 + TP_OUTER);
    const int64_t np = (o1 - o0 + TP - 1) / TP;
    for (int64_t pi = np - 1; pi >= 0; pi--) {
      const int64_t p0 = o0 + pi * TP;
      const int w = (int)std::min<int64_t>(TP, o1 - p0);
      DMB_LAUNCH(c, (k_trsm_panel<C, true>), gcols, 256, sm, N, R, p0, w, F, Linv, X);
      trsm_update<C>(c, F, N, o0, p0, p0, w, true, X, R);
    }
    trsm_update<C>(c, F, N, 0, o0, o0, (int)(o1 - o0), true, X, R);
  }
}

}  // namespace

namespace dmb {

void clear_err_word(dmb_ctx *c) {
  if (c->d_flags.p) DMB_CUDA(cudaMemsetAsync(c->d_flags.p, 0, 4, c->stream));
}

unsigned read_err_word(dmb_ctx *c) {
  unsigned e = 0;
  if (!c->d_flags.p) return 0;  // no triangular solve has run on this context
  DMB_CUDA(cudaMemcpyAsync(&e, c->d_flags.p, 4, cudaMemcpyDeviceToHost, c->stream));
  DMB_CUDA(cudaStreamSynchronize(c->stream));
  return e;
}

void nf_build(dmb_ctx *c, double cutoff, int kind) {
  double t0 = now_ms();
  const int64_t N = c->n;
  const bool f64 = c->z_prec == DMB_PREC_FP64;
  c->pc_valid = false;
  if (kind == DMB_PRECOND_NF_DIAG) {
    DevBuf &tmp = c->d_tmp[0];
    tmp.ensure(16);
    DMB_CUDA(cudaMemsetAsync(tmp.p, 0, 16, c->stream));
    c->d_dinv.ensure(sizeof(double2) * N);
    unsigned *bad = (unsigned *)(tmp.as<double>() + 1);
    if (f64) {
      DMB_LAUNCH(c, k_diag_max<double2>, 1, 1024, 0, N, c->d_Z.as<double2>(), tmp.as<double>(), bad);
      DMB_LAUNCH(c, k_diag_inv<double2>, blocks_for(N, 256), 256, 0, N, c->d_Z.as<double2>(), tmp.as<double>(),
                 c->d_dinv.as<double2>());
    } else {
      DMB_LAUNCH(c, k_diag_max<float2>, 1, 1024, 0, N, c->d_Z.as<float2>(), tmp.as<double>(), bad);
      DMB_LAUNCH(c, k_diag_inv<float2>, blocks_for(N, 256), 256, 0, N, c->d_Z.as<float2>(), tmp.as<double>(),
                 c->d_dinv.as<double2>());
    }
    double mx[2];
    DMB_CUDA(cudaMemcpyAsync(mx, tmp.p, 16, cudaMemcpyDeviceToHost, c->stream));
    DMB_CUDA(cudaStreamSynchronize(c->stream));
    unsigned hb;
    memcpy(&hb, &mx[1], 4);
    DMB_REQUIRE(hb == 0, DMB_ERR_ARGUMENT, "near-field diagonal entries must be finite");
    DMB_REQUIRE(mx[0] > 0, DMB_ERR_ARGUMENT, "cannot build a diagonal preconditioner from an all-zero diagonal");
    c->nnz_ratio = 1.0 / (double)N;
    c->pc_kind = kind;
    c->pc_prec = c->z_prec;
    c->pc_valid = true;
    c->tm.precond_ms = now_ms() - t0;
    return;
  }
  size_t esz = f64 ? sizeof(double2) : sizeof(float2);
  c->d_F.ensure(esz * N * N);
  c->d_small.ensure(65536);
  DevBuf cnt;  // view into the persistent scratch (first 8 bytes), not owned
  cnt.p = c->d_small.p;
  DMB_CUDA(cudaMemsetAsync(cnt.p, 0, 8, c->stream));
  if (!std::isfinite(cutoff) && cutoff > 0) {
    // every entry is kept: a plain device copy of Z
    DMB_CUDA(cudaMemcpyAsync(c->d_F.p, c->d_Z.p, esz * N * N, cudaMemcpyDeviceToDevice, c->stream));
    c->nnz_ratio = 1.0;
  } else {
    dim3 g(blocks_for(N, 32), blocks_for(N, 32));
    if (f64)
      DMB_LAUNCH(c, (k_nf_mask<double2, double2>), g, 256, 0, N, c->d_Z.as<double2>(), c->d_centers.as<double>(),
                 cutoff, c->d_F.as<double2>(), cnt.as<unsigned long long>());
    else
      DMB_LAUNCH(c, (k_nf_mask<float2, float2>), g, 256, 0, N, c->d_Z.as<float2>(), c->d_centers.as<double>(),
                 cutoff, c->d_F.as<float2>(), cnt.as<unsigned long long>());
    unsigned long long h_cnt = 0;
    DMB_CUDA(cudaMemcpyAsync(&h_cnt, cnt.p, 8, cudaMemcpyDeviceToHost, c->stream));
    DMB_CUDA(cudaStreamSynchronize(c->stream));
    c->nnz_ratio = ((double)h_cnt / (double)N) / (double)N;
  }
  if (f64)
    ldlt_factor(c, c->d_F.as<double2>());
  else
    ldlt_factor(c, c->d_F.as<float2>());
  c->pc_kind = kind;
  c->pc_prec = c->z_prec;
  c->pc_valid = true;
  c->tm.precond_ms = now_ms() - t0;
}

// factor a near-field matrix already written to d_F (precision of its
// storage) and make it the context's preconditioner
void nf_factor_resident(dmb_ctx *c, int kind, int precision) {
  c->pc_valid = false;
  if (precision == DMB_PREC_FP64)
    ldlt_factor(c, c->d_F.as<double2>());
  else
    ldlt_factor(c, c->d_F.as<float2>());
  c->pc_kind = kind;
  c->pc_prec = precision;
  c->pc_valid = true;
}

// what applications of the factor keep per factor, made now: a captured
// iteration replayed with a later factor does not make it
void pc_prepare_dev(dmb_ctx *c, int64_t nrhs) {
  if (c->pc_kind != DMB_PRECOND_NF_LU) return;
  if (nrhs >= 8) {  // as ldlt_solve_batched chooses
    if (c->pc_prec == DMB_PREC_MIXED && nrhs >= c->tc_min_rhs && tc_available(c))
      prepare_packed_factor(c, c->d_F.as<float2>());
    return;
  }
  if (c->pc_prec == DMB_PREC_FP64)
    prepare_block_inverses<SV, double2, double2>(c, c->d_F.as<double2>(), c->d_W.as<double2>(), c->f_inv64);
  else
    prepare_block_inverses<SV, float2, double2>(c, c->d_F.as<float2>(), c->d_W.as<double2>(), c->f_inv64);
}

void pc_apply_dev(dmb_ctx *c, double *x, int64_t nrhs) {
  DMB_REQUIRE(c->pc_valid, DMB_ERR_STATE, "no preconditioner built");
  const int64_t N = c->n;
  double2 *xd = (double2 *)x;
  if (c->pc_kind == DMB_PRECOND_NF_DIAG) {
    DMB_LAUNCH(c, k_scale_vec, blocks_for(N * nrhs, 256), 256, 0, N, nrhs, c->d_dinv.as<double2>(), xd);
    return;
  }
  if (c->pc_kind == DMB_PRECOND_NF_LU) {
    // one right-hand side at a time streams F per column; from 8 columns on
    // the panel-blocked solves read F once per sweep
    const bool batched = nrhs >= 8;
    if (c->pc_prec == DMB_PREC_FP64) {
      if (batched) ldlt_solve_batched(c, c->d_F.as<double2>(), xd, nrhs);
      else ldlt_solve(c, c->d_F.as<double2>(), xd, nrhs);
    } else {
      if (batched) ldlt_solve_batched(c, c->d_F.as<float2>(), xd, nrhs);
      else ldlt_solve(c, c->d_F.as<float2>(), xd, nrhs);
    }
    return;
  }
  if (c->pc_kind == DMB_PRECOND_LOCAL_INV || c->pc_kind == DMB_PRECOND_LEARNED || c->pc_kind == DMB_PRECOND_RING) {
    dmb::local_apply_dev(c, x, nrhs);
    return;
  }
  throw DmbError{DMB_ERR_STATE, "preconditioner kind not available"};
}

}  // namespace dmb
