// dmb_zgemm64.cu -- FP64 complex GEMM on the FP64 pipe for the plain (complex128)
// path: the Z X products of block GMRES with a complex128 Z (the zgemv of
// Krylov.gmres, one column per incidence), the trailing updates of the
// complex128 LDL^T (NearFieldPreconditioner.jl:705-715 factors the same
// matrix with UMFPACK) and the panel updates of its many-column triangular
// sweeps (:1044-1047).
//
//   Y(m, r)  =  sum_k A(m, k) B(k, r)        (OP 0)
//   Y(m, r) -=  sum_k A(m, k) B(k, r)        (OP 1)
//
// A(m, k) = A[m lda + k] (ALAY 0) or A[k lda + m] (ALAY 1); B(k, r) =
// B[r ldb + k]; Y(m, r) = Y[r ldy + m] (YLAY 0, column-major) or
// Y[m ldy + r] (YLAY 1, row-major).  LOWER keeps only r <= m (the lower
// triangle of a trailing update whose rows and columns start at the same
// index); tiles entirely above it exit at once.
//
// B200 has no FP64 tcgen05 kind, so the product runs on the FP64 matrix
// instruction (mma.sync m8n8k4, 37.0 TFLOP/s measured against 33.1 for FMA).  A
// 256-thread CTA owns a 32 x 64 complex tile, a warp 16 x 16 of it: per four k
// two A and two B fragments (one 16-byte word a lane, rows of 20 words: conflict
// free) for 16 matrix instructions, so shared memory is a quarter of the time.
// K runs in chunks of 16 through two stages filled by cp.async, three CTAs an
// SM.  The tile is this small because the products of a sweep are short: 181
// columns of a 4,720-row Z are 444 such tiles, three an SM, but 111 of 128 x 64,
// which left a quarter of the SMs idle.  Bound by the FP64 pipe.
// Measured: Z X at 4,720 x 181 1.05 ms (30.6 TFLOP/s; 1.77 ms with 128 x 64 tiles on
// FMAs), the K = 256 products of a sweep 56 us on average (169 us).
#include <algorithm>

#include "dmb_device.cuh"
#include "dmb_internal.h"

namespace {

constexpr int ZG_BM = 32, ZG_BN = 64, ZG_KC = 16, ZG_LD = ZG_KC + 4;
constexpr int ZG_A_STAGE = ZG_BM * ZG_LD, ZG_B_STAGE = ZG_BN * ZG_LD;
constexpr size_t ZG_SMEM = sizeof(double2) * 2 * (ZG_A_STAGE + ZG_B_STAGE);  // two stages: 61,440 B

// 16-byte global -> shared copy; src_bytes 0 fills the destination with zeros
// (src is then a valid address that is not read)
__device__ __forceinline__ void cp16(void *dst, const void *src, int src_bytes) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_wait_prev() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }

template <int ALAY, int YLAY, int OP, bool LOWER>
__global__ void __launch_bounds__(256, 3) k_zgemm64(int64_t M, int64_t R, int64_t K, const double2 *A, int64_t lda,
                                                    const double2 *B, int64_t ldb, double2 *Y, int64_t ldy) {
  extern __shared__ __align__(16) double2 zg_smem[];
  const int t = threadIdx.x, warp = t >> 5, l4 = t & 3, l8 = (t & 31) >> 2;
  const int64_t m0 = (int64_t)blockIdx.x * ZG_BM, n0 = (int64_t)blockIdx.y * ZG_BN;
  if (LOWER && n0 > m0 + ZG_BM - 1) return;
  // chunk of K from k0 into stage s: two A and four B elements per thread
  auto issue = [&](int64_t k0, int s) {
    double2 *As = zg_smem + s * ZG_A_STAGE;
    double2 *Bs = zg_smem + 2 * ZG_A_STAGE + s * ZG_B_STAGE;
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const int e = t + 256 * u;
      const int mm = ALAY == 0 ? e >> 4 : e & 31, kk = ALAY == 0 ? e & 15 : e >> 5;
      const int64_t m = m0 + mm, k = k0 + kk;
      const bool in = m < M && k < K;
      cp16(As + mm * ZG_LD + kk, in ? (ALAY == 0 ? A + m * lda + k : A + k * lda + m) : A, in ? 16 : 0);
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int e = t + 256 * u;
      const int rr = e >> 4, kk = e & 15;
      const int64_t r = n0 + rr, k = k0 + kk;
      const bool in = r < R && k < K;
      cp16(Bs + rr * ZG_LD + kk, in ? B + r * ldb + k : B, in ? 16 : 0);
    }
  };
  const int wm = 16 * (warp & 1), wn = 16 * (warp >> 1);
  double re[2][2][2], im[2][2][2];
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 2; j++) re[i][j][0] = re[i][j][1] = im[i][j][0] = im[i][j][1] = 0.0;
  const int64_t nch = (K + ZG_KC - 1) / ZG_KC;
  if (nch > 0) issue(0, 0);
  cp_commit();
  for (int64_t ch = 0; ch < nch; ch++) {
    if (ch + 1 < nch) issue((ch + 1) * ZG_KC, (int)((ch + 1) & 1));
    cp_commit();
    cp_wait_prev();  // chunk ch has landed (this thread's copies)
    __syncthreads();
    const double2 *As = zg_smem + (ch & 1) * ZG_A_STAGE + (wm + l8) * ZG_LD + l4;
    const double2 *Bs = zg_smem + 2 * ZG_A_STAGE + (ch & 1) * ZG_B_STAGE + (wn + l8) * ZG_LD + l4;
#pragma unroll
    for (int kk = 0; kk < ZG_KC; kk += 4) {
      double2 a[2], b[2];
#pragma unroll
      for (int i = 0; i < 2; i++) a[i] = As[8 * i * ZG_LD + kk];
#pragma unroll
      for (int j = 0; j < 2; j++) b[j] = Bs[8 * j * ZG_LD + kk];
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 2; j++) zmma(re[i][j], im[i][j], a[i], b[j]);
    }
    __syncthreads();  // stage ch & 1 is refilled by the next iteration's issue
  }
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const int64_t m = m0 + wm + 8 * i + l8;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const int64_t r = n0 + wn + 8 * j + 2 * l4 + u;
        if (r >= R || (LOWER && r > m)) continue;
        double2 *p = YLAY == 0 ? Y + r * ldy + m : Y + m * ldy + r;
        const double2 v = make_double2(re[i][j][u], im[i][j][u]);
        *p = OP == 0 ? v : csub(*p, v);
      }
  }
}

template <int ALAY, int YLAY, int OP, bool LOWER>
void launch(dmb_ctx *c, int64_t M, int64_t R, int64_t K, const double2 *A, int64_t lda, const double2 *B, int64_t ldb,
            double2 *Y, int64_t ldy) {
  if (M <= 0 || R <= 0) return;
  raise_smem(c, k_zgemm64<ALAY, YLAY, OP, LOWER>, ZG_SMEM);
  dim3 g((unsigned)((M + ZG_BM - 1) / ZG_BM), (unsigned)((R + ZG_BN - 1) / ZG_BN));
  DMB_LAUNCH(c, (k_zgemm64<ALAY, YLAY, OP, LOWER>), g, 256, ZG_SMEM, M, R, K, A, lda, B, ldb, Y, ldy);
}

}  // namespace

namespace dmb {

// Z X and the sweep updates are timed as kernel family 4 (8 flops per
// complex MAC); the factor's updates are timed by their caller (family 2).
void zgemm64_zx(dmb_ctx *c, const double2 *Z, const double2 *X, double2 *Y, int64_t N, int64_t R) {
  kt_begin(c);
  launch<0, 0, 0, false>(c, N, R, N, Z, N, X, N, Y, N);  // K = N = 0 still writes Y = 0
  kt_end(c, 8.0 * (double)N * (double)N * (double)R, 4);
}

void zgemm64_sub(dmb_ctx *c, bool a_transposed, int64_t M, int64_t R, int64_t K, const double2 *A, int64_t lda,
                 const double2 *B, int64_t ldb, double2 *Y, int64_t ldy) {
  if (K <= 0) return;
  kt_begin(c);
  if (a_transposed)
    launch<1, 0, 1, false>(c, M, R, K, A, lda, B, ldb, Y, ldy);
  else
    launch<0, 0, 1, false>(c, M, R, K, A, lda, B, ldb, Y, ldy);
  kt_end(c, 8.0 * (double)M * (double)R * (double)K, 4);
}

void zgemm64_lower_update(dmb_ctx *c, int64_t M, int64_t C, int64_t K, const double2 *W, int64_t ldw,
                          const double2 *Lrows, int64_t ldl, double2 *F, int64_t ldf) {
  if (K <= 0) return;
  launch<0, 1, 1, true>(c, M, C, K, W, ldw, Lrows, ldl, F, ldf);
}

}  // namespace dmb
