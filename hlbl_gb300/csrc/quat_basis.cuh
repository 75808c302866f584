// quat_basis.cuh -- the block-diagonal form of pass 2's contraction
//   F[nu][lam] = Re sum_{p,q} D[p][q] M[q][p],  M = Gt_lam dz Gt_nu   (per j, mu)
// (bt_build_kernel's M, with the gamma insertions written out).
//
// gamma_mu gamma_5 maps the spin pair (0, 1) of one chirality to that of the
// other, and between the pairs every gamma is a unit of the quaternions
//   q_0 = 1, q_1 = i sigma_1, q_2 = i sigma_2, q_3 = i sigma_3
// up to a sign. So for each chirality block chi = (chi_p, chi_q) of D and
// each pair of colours, F depends on the 2 x 2 spin matrices
//   X = D[(2 chi_p + i, c_p)][(2 chi_q + k, c_q)],
//   Z = dz[(2 (1-chi_q) + i, c_q)][(2 (1-chi_p) + k, c_p)]
// only through their quaternion components x_b, z_a (times two: X00 + X11,
// -i (X01 + X10), X01 - X10, -i (X00 - X11)), and q_lam q_a q_nu is a unit:
//   F[nu][lam] = sum_chi sum_{a,b} t_chi[nu][lam][a][b] Re(sum_colours x_b z_a) / 2
// with t = 0 unless nu ^ lam ^ a ^ b = 0, else a sign. Per (j, mu, b, chi) that
// is a dot of length 18 (nine colour pairs, re and im) with four columns a, in
// place of one of length 288 with sixteen columns (nu, lam): a quarter of the
// multiply-adds, for the same F. The signs of the four blocks differ in nu and
// lam, so the blocks' results are weighted apart (class_sums below).
#pragma once

#include "hlbl_device.cuh"

namespace hg {
namespace quat {

constexpr int kBlk = 4;              // chirality blocks, 2 chi_p + chi_q
constexpr int kKb = 18;              // (c_p, c_q, re/im) of a block
constexpr int kCol = 40;             // (j, a)
constexpr int kLen = kBlk * kKb * kCol;  // dz in this form, per flavour: [blk][k][j*4 + a]

// entry (r, c) of q_u as a power of i, or -1 for zero
__host__ __device__ constexpr int unit_ph(int u, int r, int c) {
  return u == 0 ? (r == c ? 0 : -1)
       : u == 1 ? (r != c ? 1 : -1)
       : u == 2 ? (r != c ? (r == 0 ? 0 : 2) : -1)
       : (r == c ? (r == 0 ? 1 : 3) : -1);
}
// t of the block chi = (0, 0): the sum over p, q of the spin factors, over two
__host__ __device__ constexpr int base_sign(int nu, int lam, int a, int b) {
  int re = 0;
  for (int p = 0; p < 2; ++p)
    for (int q = 0; q < 2; ++q) {
      int const c = gg5_src(lam, q), bb = gg5_src(nu, p);  // both in the other pair
      int const x = unit_ph(b, p, q), z = unit_ph(a, c - 2, bb - 2);
      if (x < 0 || z < 0) continue;
      int const ph = (x + z + gg5_ph(nu, p) + gg5_ph(lam, c)) & 3;
      re += ph == 0 ? 1 : (ph == 2 ? -1 : 0);
    }
  return re / 2;
}
// sign bits of t_(0,0)[m][m ^ a ^ b][a][b], m = 0..3 (1: negative)
__host__ __device__ constexpr unsigned base_mask(int a, int b) {
  unsigned v = 0;
  for (int m = 0; m < 4; ++m) v |= base_sign(m, m ^ a ^ b, a, b) < 0 ? 1u << m : 0u;
  return v;
}
// sixteen masks of four bits, (a, b) at bit 4 (4 a + b)
__host__ __device__ constexpr unsigned long long base_masks() {
  unsigned long long v = 0;
  for (int a = 0; a < 4; ++a)
    for (int b = 0; b < 4; ++b) v |= (unsigned long long)base_mask(a, b) << (4 * (4 * a + b));
  return v;
}
constexpr unsigned long long kBaseMasks = base_masks();

__device__ __forceinline__ double flip(double v, unsigned neg) {
  return __hiloint2double(__double2hiint(v) ^ (int)(neg << 31), __double2loint(v));
}
__device__ __forceinline__ float flip(float v, unsigned neg) {
  return __uint_as_float(__float_as_uint(v) ^ (neg << 31));
}

// sum_{nu, lam} t_chi[nu][lam][a][b] c[nu][lam] for the four blocks chi =
// (0,0), (0,1), (1,0), (1,1), from the four c[m] = c[nu = m][lam = m ^ kappa]
// of the class kappa = a ^ b. The blocks differ by a sign of nu, of lam or of
// both: t_chi = (-1)^(chi_p + chi_q) s_nu^chi_p s_lam^chi_q t_(0,0), s = (+,-,-,-).
template <typename T>
__device__ __forceinline__ void class_sums(const T c[4], int kappa, int a, int b, T out[4]) {
  unsigned const m = (unsigned)(kBaseMasks >> (4 * (4 * a + b)));
  T e[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) e[i] = flip(c[i], (m >> i) & 1u);
  if (kappa == 0) {
    T const r = e[1] + e[2] + e[3];
    out[0] = out[3] = e[0] + r;
    out[1] = out[2] = r - e[0];
  } else {
    T const ek = kappa == 1 ? e[1] : (kappa == 2 ? e[2] : e[3]);
    T const u = e[0] + ek, w = e[0] - ek;
    T const v = kappa == 1 ? e[2] + e[3] : (kappa == 2 ? e[1] + e[3] : e[1] + e[2]);
    out[0] = u + v;
    out[1] = v + w;
    out[2] = v - w;
    out[3] = v - u;
  }
}

// twice the quaternion components of the 2 x 2 complex matrix (x00, x01, x10, x11)
template <typename T>
__device__ __forceinline__ void components(const T x00[2], const T x01[2], const T x10[2], const T x11[2], T c[4][2]) {
  c[0][0] = x00[0] + x11[0]; c[0][1] = x00[1] + x11[1];
  c[1][0] = x01[1] + x10[1]; c[1][1] = -(x01[0] + x10[0]);
  c[2][0] = x01[0] - x10[0]; c[2][1] = x01[1] - x10[1];
  c[3][0] = x00[1] - x11[1]; c[3][1] = x11[0] - x00[0];
}

}  // namespace quat
}  // namespace hg
