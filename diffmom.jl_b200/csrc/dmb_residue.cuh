// dmb_residue.cuh -- what the int8 residue products share: the moduli and the
// Chinese-remainder constants, the reduction of int32 sums, the 96-bit
// fraction sums, and the int8 MMA of a 128 x 256 tile.  The scheme is that of
// dmb_ozaki.cu (its head has the derivation and the published source).
#pragma once
#include <cmath>

#include "dmb_tcgen05.cuh"

namespace dmb_tc {

constexpr int OZ_BM = 128, OZ_BN = 256, OZ_BK = 128;  // BK in bytes (= int8 K elements)
// D s32, A/B signed int8, K-major, N = 256, M = 128
constexpr uint32_t OZ_IDESC = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(OZ_BN >> 3) << 17) |
                              ((uint32_t)(OZ_BM >> 4) << 24);

// pairwise coprime moduli, largest first (255 = 3 5 17, 253 = 11 23,
// 247 = 13 19, 217 = 7 31, the rest prime): the first 13 make the products of
// a complex64 Z (M ~ 2^102.5), all 16 those of complex128 operands (2^125.4)
constexpr int OZ_NMOD = 13, OZ_NMOD64 = 16;
constexpr int OZ_MODULI[OZ_NMOD64] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193};

// v mod m in [0, m) for an int8-product sum |v| <= 2^31 - 2^14 and
// 193 <= m <= 256, in integer arithmetic: u = v + moff (moff = m
// floor(2^31 / m), so 0 < u < 2^32 and u = v mod m), q = floor(u mmul /
// 2^39) with mmul = ceil(2^39 / m) is floor(u / m) or one more (the error of
// u mmul / 2^39 is below u / 2^39 < 2^-7), one correction.
__device__ __forceinline__ unsigned oz_mod(int v, unsigned m, unsigned mmul, unsigned moff) {
  const unsigned u = (unsigned)v + moff;
  const unsigned q = __umulhi(u, mmul) >> 7;
  const int r = (int)(u - q * m);
  return (unsigned)(r < 0 ? r + (int)m : r);
}

// Global accesses to the residue planes marked evict-last in L2: a CTA's
// planes (416 KB) are read back at its tile's last modulus, while the int8
// operand planes stream through L2 once per product.
__device__ __forceinline__ uint64_t l2_evict_last_policy() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint4 ld_keep4(const uint4 *a, uint64_t pol) {
  uint4 v;
  asm volatile("ld.global.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(a), "l"(pol));
  return v;
}
__device__ __forceinline__ void st_keep4(uint4 *a, uint4 v, uint64_t pol) {
  asm volatile("st.global.L2::cache_hint.v4.u32 [%0], {%1, %2, %3, %4}, %5;" ::"l"(a), "r"(v.x), "r"(v.y),
               "r"(v.z), "r"(v.w), "l"(pol)
               : "memory");
}

__device__ __forceinline__ void umma_i8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(OZ_IDESC), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// S = sum over the 16 residues packed in p (bytes, element q in byte q) of
// r_q f, f = fh 2^32 + fl, accumulated as th 2^32 + tl (tl < 2^44 for up to
// 16 terms, so no carry is lost before the final fold)
__device__ __forceinline__ void oz_frac_add(const uint4 p, unsigned long long fh, unsigned long long fl,
                                            unsigned long long (&th)[16], unsigned long long (&tl)[16]) {
  const unsigned w[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
  for (int q = 0; q < 16; q++) {
    const unsigned long long u = (w[q >> 2] >> (8 * (q & 3))) & 0xffu;
    tl[q] += u * fl;
    th[q] += u * fh;
  }
}

// Chinese-remainder constants of the first nm moduli
struct CrtConst {
  unsigned __int128 M = 1;
  double log2M = 0;
  unsigned long long frac[OZ_NMOD64];
  unsigned fraclo[OZ_NMOD64];
};
inline CrtConst crt_const(int nm) {
  CrtConst k;
  for (int i = 0; i < nm; i++) {
    k.M *= (unsigned)OZ_MODULI[i];
    k.log2M += std::log2((double)OZ_MODULI[i]);
  }
  for (int i = 0; i < nm; i++) {
    const int mi = OZ_MODULI[i];
    int Mi = 1;  // (M / m_i) mod m_i
    for (int j = 0; j < nm; j++)
      if (j != i) Mi = (Mi * (OZ_MODULI[j] % mi)) % mi;
    int y = 1;
    while ((Mi * y) % mi != 1) y++;  // m_i <= 256: direct search
    const unsigned __int128 f = (((unsigned __int128)y << 96) + (unsigned)(mi / 2)) / (unsigned)mi;  // < 2^96
    k.frac[i] = (unsigned long long)(f >> 32);
    k.fraclo[i] = (unsigned)(f & 0xffffffffu);
  }
  return k;
}
inline bool crt_fits(int64_t K, int e, const CrtConst &k) {  // K 2^e < M / 2
  return e >= 0 && e <= 114 && ((unsigned __int128)K << (e + 1)) < k.M;  // K < 2^13 at e = 114, 2^18 below 100
}

}  // namespace dmb_tc
