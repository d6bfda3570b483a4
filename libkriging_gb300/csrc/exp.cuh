// exp.cuh -- exp(x) for the covariance kernels, in ten FP64 operations.
//
// Tang's table-driven exponential (ACM TOMS 15(2), 1989): x = (64 q + i) ln2 / 64 + r with |r| <= ln2 / 128, and
// exp(x) = 2^q T_i (1 + r + r^2 / 2 + ... + r^5 / 120), T_i = 2^(i / 64) from a table of 64 doubles; the dropped term is
// below 2^-54.  FP64 issue bounds every kernel that takes an exponential per pair (19 clocks per warp instruction and
// SM, a 64-clock latency each); CUDA's exp takes 17 of them.  Within 1.25 units in the last place (0.32 on average).
#pragma once
#include <cuda_runtime.h>

namespace lkg {

__device__ __constant__ const double kExpTable[64] = {
    0x1.0000000000000p+0, 0x1.02c9a3e778061p+0, 0x1.059b0d3158574p+0, 0x1.0874518759bc8p+0,
    0x1.0b5586cf9890fp+0, 0x1.0e3ec32d3d1a2p+0, 0x1.11301d0125b51p+0, 0x1.1429aaea92de0p+0,
    0x1.172b83c7d517bp+0, 0x1.1a35beb6fcb75p+0, 0x1.1d4873168b9aap+0, 0x1.2063b88628cd6p+0,
    0x1.2387a6e756238p+0, 0x1.26b4565e27cddp+0, 0x1.29e9df51fdee1p+0, 0x1.2d285a6e4030bp+0,
    0x1.306fe0a31b715p+0, 0x1.33c08b26416ffp+0, 0x1.371a7373aa9cbp+0, 0x1.3a7db34e59ff7p+0,
    0x1.3dea64c123422p+0, 0x1.4160a21f72e2ap+0, 0x1.44e086061892dp+0, 0x1.486a2b5c13cd0p+0,
    0x1.4bfdad5362a27p+0, 0x1.4f9b2769d2ca7p+0, 0x1.5342b569d4f82p+0, 0x1.56f4736b527dap+0,
    0x1.5ab07dd485429p+0, 0x1.5e76f15ad2148p+0, 0x1.6247eb03a5585p+0, 0x1.6623882552225p+0,
    0x1.6a09e667f3bcdp+0, 0x1.6dfb23c651a2fp+0, 0x1.71f75e8ec5f74p+0, 0x1.75feb564267c9p+0,
    0x1.7a11473eb0187p+0, 0x1.7e2f336cf4e62p+0, 0x1.82589994cce13p+0, 0x1.868d99b4492edp+0,
    0x1.8ace5422aa0dbp+0, 0x1.8f1ae99157736p+0, 0x1.93737b0cdc5e5p+0, 0x1.97d829fde4e50p+0,
    0x1.9c49182a3f090p+0, 0x1.a0c667b5de565p+0, 0x1.a5503b23e255dp+0, 0x1.a9e6b5579fdbfp+0,
    0x1.ae89f995ad3adp+0, 0x1.b33a2b84f15fbp+0, 0x1.b7f76f2fb5e47p+0, 0x1.bcc1e904bc1d2p+0,
    0x1.c199bdd85529cp+0, 0x1.c67f12e57d14bp+0, 0x1.cb720dcef9069p+0, 0x1.d072d4a07897cp+0,
    0x1.d5818dcfba487p+0, 0x1.da9e603db3285p+0, 0x1.dfc97337b9b5fp+0, 0x1.e502ee78b3ff6p+0,
    0x1.ea4afa2a490dap+0, 0x1.efa1bee615a27p+0, 0x1.f50765b6e4540p+0, 0x1.fa7c1819e90d8p+0,
};

// the table in shared memory, filled by the block's threads (lanes read different entries); a barrier must follow
template <int NTH>
__device__ __forceinline__ void exp_table_fill(double* tab) {
  for (int i = threadIdx.x; i < 64; i += NTH) tab[i] = kExpTable[i];
}

// exp(x); outside [-708, 2) and for NaN through the library's exp
__device__ __forceinline__ double exp_tab(double x, const double* tab) {
  const int hi = __double2hiint(x);
  if ((unsigned)hi > 0xC0862000u || (hi >= 0x40000000)) return exp(x);
  const double t = fma(x, 0x1.71547652b82fep+6, 6755399441055744.0);  // 64 / ln2; 1.5 2^52 leaves the rounded integer in the low word
  const int n = __double2loint(t);
  const double k = t - 6755399441055744.0;
  double r = fma(k, -0x1.62e42fef80000p-7, x);  // ln2 / 64, 34 bits: the product with |k| < 2^17 is exact
  r = fma(k, -0x1.1cf79abc9e3b4p-42, r);
  double p = fma(r, 1.0 / 120.0, 1.0 / 24.0);
  p = fma(r, p, 1.0 / 6.0);
  p = fma(r, p, 0.5);
  p = fma(r * r, p, r);
  const double T = tab[n & 63];
  const double e = fma(T, p, T);
  return __hiloint2double(__double2hiint(e) + ((n >> 6) << 20), __double2loint(e));
}

}  // namespace lkg
