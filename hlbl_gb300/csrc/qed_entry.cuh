// qed_entry.cuh -- entries of the closed-form stand-in tensor in FP64 from
// tabulated factors.
#pragma once

#include <cuda_runtime.h>

#include "contract_kernels.cuh"

namespace hg {

// v, or its negative (bit 0 of neg), without an FP64 instruction
__device__ __forceinline__ double flip_sign(double v, unsigned neg) {
  return __hiloint2double(__double2hiint(v) ^ (int)(neg << 31), __double2loint(v));
}

constexpr int kQedTab = 63;  // factors of the tensor's terms per (site, evaluation)

// Factor i of the evaluation with arguments a, b and weights w.
// tab: w0 a[4] | w1 b[4] | w2 (a-b)[4] | w3 (a_r b_s - a_s b_r)[6] | (a+b)[4] |
//      w4 a[4] | b_i b_j [16] | w5 b[4] | a_i a_j [16] | 0
__device__ __forceinline__ double qed_tab_value(int i, const double* a, const double* b, const double* w) {
  if (i < 4) return w[0] * a[i];
  if (i < 8) return w[1] * b[i - 4];
  if (i < 12) return w[2] * (a[i - 8] - b[i - 8]);
  if (i < 18) {
    int const r = comb_rho(i - 12), g = comb_sigma(i - 12);
    return w[3] * (a[r] * b[g] - a[g] * b[r]);
  }
  if (i < 22) return a[i - 18] + b[i - 18];
  if (i < 26) return w[4] * a[i - 22];
  if (i < 42) return b[(i - 26) >> 2] * b[(i - 26) & 3];
  if (i < 46) return w[5] * b[i - 42];
  if (i < 62) return a[(i - 46) >> 2] * a[(i - 46) & 3];
  return 0.0;
}

// One entry kerv[k][mu][nu][lam] of the stand-in (qed_entry_t's six terms)
// from the tabulated factors: two adds and three multiply-adds whatever the
// indices (terms that vanish are selected to zero on the integer pipe; with
// branches the lanes of a warp, which hold different entries, issue all
// eleven).
__device__ __forceinline__ double qed_entry_tab(const double* __restrict__ tab, int k, int r, int s, int mu, int nu, int lam) {
  double const t0 = mu == r && nu == s ? tab[lam] : (mu == s && nu == r ? flip_sign(tab[lam], 1u) : 0.0);
  double const t1 = mu == r && lam == s ? tab[4 + nu] : (mu == s && lam == r ? flip_sign(tab[4 + nu], 1u) : 0.0);
  double const t2 = nu == r && lam == s ? tab[8 + mu] : (nu == s && lam == r ? flip_sign(tab[8 + mu], 1u) : 0.0);
  double const f3 = mu == nu ? tab[12 + k] : 0.0;
  double const f4 = mu == s ? tab[22 + r] : (mu == r ? flip_sign(tab[22 + s], 1u) : 0.0);
  double const f5 = lam == s ? tab[42 + r] : (lam == r ? flip_sign(tab[42 + s], 1u) : 0.0);
  double v = t0 + t1 + t2;
  v = fma(f3, tab[18 + lam], v);
  v = fma(f4, tab[26 + 4 * nu + lam], v);
  return fma(f5, tab[46 + 4 * mu + nu], v);
}

}  // namespace hg
