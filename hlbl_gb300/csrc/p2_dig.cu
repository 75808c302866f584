// p2_dig.cu -- the FP64 pass 2 (ker_4pt_contraction, cuda_lattice.cu:277-484)
// without FP64 products: the spin-block products in 64-bit integers and the
// contraction as exact products of digits on the tensor cores.
//
// What bounds the direct form is the FP64 pipe (two lanes per SM and cycle
// here): 14.9 k multiply-adds per site and flavour for D_mu and 46.1 k for the
// contraction even in the block-diagonal form of p2_f64.cu. Here
//   D_mu   the blocks' values as 58-bit integers of a common exponent per site,
//          two limbs of 29 bits, three 32 x 32 -> 64-bit integer multiply-adds
//          per product (the product of the low limbs, below 2^-56 of the
//          largest product, is dropped): sums of 24 such products stay below
//          2^61, so nothing is rounded before the one rounding to 57 bits (with
//          the sign) below the site's largest |D|;
//   F = D Bt  D and Bt (per column) as eight balanced digits, seven of base 128
//          and a top one of up to 128, in FP16; digit products with i + j <= 7
//          (i = 0 the top) are accumulated by weight in eight FP32 accumulators
//          in TMEM: each is an integer below 2^24 (288 k; at most two products of
//          128 x 64 and six of 64 x 64), hence exact; the weights are put
//          together in 64-bit integers.
// The only roundings are those of the inputs to fixed point (2^-58 of the
// site's largest component), of D and Bt (2^-57 of the site's and the column's
// largest), the dropped products (i + j > 7: below 2^-53 of a typical F) and F's
// conversion; the FP64 form rounds at 2^-53 of every partial sum. Roundings with a
// mean add up over the sites where random ones do not, so D's is to nearest even,
// and the mean of the products of weight 8 (D's lower digits, -64 to 63, have the
// mean -1/2) is added per column.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "contract_kernels.cuh"
#include "hlbl_gb300.h"
#include "hlbl_internal.h"
#include "fixed_point.cuh"
#include "p2_dig.h"
#include "qed_entry.cuh"
#include "tc_ops.cuh"

namespace hg {
namespace dig {

using ll = long long;
using ull = unsigned long long;

constexpr int kSites = 32;            // sites per tile
constexpr int kRows = 4 * kSites;     // rows (mu, site) of a tile: M of the MMA
constexpr int kChunks = kBtK / 16;    // MMA steps of K = 16
constexpr int kDig = 8;               // digits of a value
constexpr int kAcc = kDig;            // accumulators: weights i + j
constexpr int kParts = 3;             // the 160 columns in parts of 64, 64, 32 (eight accumulators in 512 TMEM columns)
constexpr int kMaxTiles = 304;        // tiles of a batch
constexpr int kMaxSites = kMaxTiles * kSites;
// words of a tile and flavour: [chunk][k / 8][row][k % 8 / 2]
constexpr int kTileWords = kChunks * 2 * kRows * 4;
// digits are stored with 64 (the top: 128) added to each: D's as two values'
// (re, im) 16-bit halves per word, digit 2 w + 1 in bits 0-6 and digit 2 w from
// bit 7 (word w = 0..3; the top digit's nine bits: 0 to 256), as the MMA's A wants
// neighbouring k side by side
constexpr ull kBias = 64ull * ((1ull << 49) - 1) / 127 + (128ull << 49);
constexpr int kZeroRow = -20000;      // row exponent of a row of Bt of zeros only
constexpr int kRowExp = 24;           // per flavour: of Y's rows p, of S's rows q

__host__ __device__ constexpr int part_n0(int p) { return 64 * p; }
__host__ __device__ constexpr int part_n(int p) { return p < 2 ? 64 : 32; }
// bytes before part p's digits of Bt, and of one of its chunks
__host__ __device__ constexpr int part_base(int p) { return part_n0(p) * kChunks * kDig * 32; }
__host__ __device__ constexpr int part_chunk(int p) { return part_n(p) * kDig * 32; }
constexpr size_t kBtBytes = (size_t)kBtN * kChunks * kDig * 32;  // per flavour

// ---- Bt's digits ---------------------------------------------------------------
// Entry (p, q) of column n = (j, nu, lam) of Bt (bt_build_kernel's values), complex,
// from pass 1's sums dz or from sums with the gammas inserted.
__device__ __forceinline__ void bt_entry(const double* __restrict__ dz, const double* __restrict__ g_dzu,
                                         const double* __restrict__ g_dzsu, int n, int p, int q, double& re, double& im) {
  int const lam = n & 3, nu = (n >> 2) & 3, j = n >> 4;
  int const s2 = gg5_src(lam, q / 3), sp = p / 3;  // an involution
  int const ia = 3 * s2 + q % 3;
  if (dz != nullptr) {
    const double* v = dz + ((j * 12 + ia) * 12 + 3 * gg5_src(nu, sp) + p % 3) * 2;
    mul_iph((gg5_ph(lam, s2) + gg5_ph(nu, sp)) & 3, v[0], v[1], re, im);
  } else {
    const double* g = (j < 6 ? g_dzu + (size_t)j * 1152 : g_dzsu + (size_t)(j - 6) * 1152) + ((nu * 12 + ia) * 12 + p) * 2;
    mul_iph(gg5_ph(lam, s2), g[0], g[1], re, im);
  }
}

// Powers of two that take the scale of the rows out of Bt and into D, so that a
// D's fixed-point error is measured by what the value contributes (rows, e.g. of
// one colour, may differ in scale): Bt(p, q) 2^(-b_p - c_q), Y_p 2^b_p, S_q 2^c_q.
constexpr int kRowThreads = 576;
__global__ void __launch_bounds__(kRowThreads)
brow_kernel(const double* __restrict__ dz, const double* __restrict__ g_dzu, const double* __restrict__ g_dzsu,
            int* __restrict__ rowexp) {
  __shared__ int s_e[144], s_b[12];
  int const fl = blockIdx.x, t = threadIdx.x, pq = t >> 2;
  if (dz != nullptr) dz += (size_t)fl * kDzLen;
  int m = kZeroExp;
  // over all columns (j, nu, lam) the entries are those of the images' spins: (p, q)'s
  // colours with every pair of spins (a, b), or of each nu with every spin b of q
  int const p = pq / 12, q = pq % 12;
#pragma unroll 10
  for (int n = t & 3; n < kBtN; n += 4) {
    int const j = n >> 4, a = (n >> 2) & 3, b = n & 3;
    const double* v = dz != nullptr ? dz + ((j * 12 + 3 * a + q % 3) * 12 + 3 * b + p % 3) * 2
                                    : (j < 6 ? g_dzu + (size_t)j * 1152 : g_dzsu + (size_t)(j - 6) * 1152) +
                                          ((a * 12 + 3 * b + q % 3) * 12 + p) * 2;
    double2 const z = *reinterpret_cast<const double2*>(v);
    m = max(m, max(exp_of(z.x, 0), exp_of(z.y, 0)));
  }
  m = max(m, __shfl_xor_sync(0xffffffffu, m, 1));
  m = max(m, __shfl_xor_sync(0xffffffffu, m, 2));
  if ((t & 3) == 0) s_e[pq] = min(m, 2047);
  __syncthreads();
  if (t < 12) {
    int b = kZeroExp;
    for (int q = 0; q < 12; ++q) b = max(b, s_e[t * 12 + q]);
    s_b[t] = b == kZeroExp ? kZeroRow : b;
    rowexp[fl * kRowExp + t] = s_b[t];
  }
  __syncthreads();
  if (t < 12) {
    int c = kZeroExp;
    for (int p = 0; p < 12; ++p)
      if (s_e[p * 12 + t] != kZeroExp) c = max(c, s_e[p * 12 + t] - s_b[p]);
    rowexp[fl * kRowExp + 12 + t] = c == kZeroExp ? kZeroRow : c;
  }
}

// Column n's digits, k = 2 (12 p + q) + e; em[fl][n]: the exponent of its largest value;
// corr[fl][n]: the mean of the dropped products of weight 8, in units of weight 7.
__global__ void __launch_bounds__(kBtK)
bdig_build_kernel(const double* __restrict__ dz, const double* __restrict__ g_dzu, const double* __restrict__ g_dzsu,
                  const int* __restrict__ rowexp, unsigned char* __restrict__ bt, int* __restrict__ em,
                  int* __restrict__ corr) {
  __shared__ int s_em, s_sum;
  int const n = blockIdx.x, fl = blockIdx.y, k = threadIdx.x;
  int const e = k & 1, q = (k >> 1) % 12, p = k / 24;
  if (dz != nullptr) dz += (size_t)fl * kDzLen;
  double re, im;
  bt_entry(dz, g_dzu, g_dzsu, n, p, q, re, im);
  double const x = e == 0 ? re : -im;
  int const r = -rowexp[fl * kRowExp + p] - rowexp[fl * kRowExp + 12 + q];
  if (k == 0) {
    s_em = kZeroExp;
    s_sum = 0;
  }
  __syncthreads();
  atomicMax(&s_em, exp_of(x, r));
  __syncthreads();
  int const m = s_em;
  if (k == 0) em[fl * kBtN + n] = m;
  ull const w = (ull)to_fixed<3>(x, r, m) + kBias;
  int const part = n < 128 ? n >> 6 : 2, np = part_n(part);
  unsigned char* out = bt + (size_t)fl * kBtBytes + part_base(part) + (size_t)(k >> 4) * part_chunk(part) +
                       (((k >> 3) & 1) * kDig * np + n - part_n0(part)) * 16 + (k & 7) * 2;
  int sum = 0;
#pragma unroll
  for (int i = 0; i < kDig; ++i) {
    int const u = (int)(w >> (7 * (kDig - 1 - i))) & (i == 0 ? 0x1FF : 0x7F), b = u - (i == 0 ? 128 : 64);
    *reinterpret_cast<__half*>(out + (size_t)i * np * 16) = __int2half_rn(b);
    if (i > 0) sum += b;
  }
  sum = __reduce_add_sync(0xffffffffu, sum);
  if ((k & 31) == 0) atomicAdd(&s_sum, sum);
  __syncthreads();
  if (k == 0) corr[fl * kBtN + n] = (int)rintf(-0.5f / 128.f * (float)s_sum);
}

// ---- D's words -----------------------------------------------------------------
constexpr int kTS = 4;                  // sites per CTA
constexpr int kDThreads = 160;          // of a CTA of either role; here 144 threads (p, q) at work
constexpr int kRowD = kTS * 24 + 2;     // staged row: 16 bytes of padding against bank conflicts

// The sites s_begin + 4 block ... of the batch, flavour f0 + fl
// (independent CTAs of 160 threads hide each other's copies and barriers: 188 -> 170 us
// at 8,192 sites against 320 threads for both flavours). words[tile][fl][kTileWords],
// esc[fl][site]: D (its rows scaled by rowexp) = integer 2^esc.
struct __align__(128) DSmem {
  double stage[24][kRowD];
  uint64_t bar;
  int em[2][kTS];
  uint32_t top[2][5][2];
};
__device__ __forceinline__ void
dform_cta(DSmem& sm, const double* __restrict__ y, const double* __restrict__ src, const Geometry& geo, int f0, int fl,
          int nf, int block, ll s_begin, const int* __restrict__ rowexp, uint4* __restrict__ words, int* __restrict__ esc,
          int* __restrict__ err) {
  double (*const stage)[kRowD] = sm.stage;
  uint64_t& s_bar = sm.bar;
  int (*const s_em)[kTS] = sm.em;
  uint32_t (*const s_or)[5][2] = sm.top;
  int const t = threadIdx.x, l0 = kTS * block;
  ll const s0 = s_begin + l0;
  int const nvalid = (int)min((ll)kTS, geo.V - s0);
  if (t == 0) {
    mbar_init(&s_bar, 1);
    fence_mbar_init();
  }
  if (t < 2 * kTS) (&s_em[0][0])[t] = kZeroExp;
  __syncthreads();
  if (t == 0) {
    // S = src at flavour 1-f, Y = y at flavour f, f = f0 + fl; rows [S | Y][12]
    uint32_t const bytes = (uint32_t)nvalid * 192u;
    mbar_arrive_expect_tx(&s_bar, bytes * 24);
    for (int row = 0; row < 24; ++row) {
      int const f = row < 12 ? 1 - f0 - fl : f0 + fl;
      bulk_g2s(stage[row], (row < 12 ? src : y) + ((size_t)(f * 12 + row % 12) * geo.V + s0) * 24, bytes, &s_bar);
    }
  }
  bool const ok = mbar_wait(&s_bar, 0);
  if (__syncthreads_or(!ok)) {
    // the copies land before the CTA exits (bounded, as everything else)
    if (t == 0) {
      if (err) atomicExch(err, kErrWaitTimeout);
      mbar_wait(&s_bar, 0);
    }
    return;
  }
  {
    // to fixed point in place: (site, S or Y) by 20 threads each
    constexpr int kPer = kDThreads / (2 * kTS), kVals = (288 + kPer - 1) / kPer;
    int const g = t / kPer, i0 = t % kPer, s = g % kTS, which = g / kTS;
    double (*const rows)[kRowD] = &stage[which * 12];
    const int* const rx = rowexp + fl * kRowExp + (which == 0 ? 12 : 0);  // S: of rows q, Y: of rows p
    double v[kVals];
    int m = kZeroExp;
    if (s < nvalid) {
#pragma unroll
      for (int i = 0; i < kVals; ++i) {
        int const idx = i0 + i * kPer;
        v[i] = idx < 288 ? rows[idx / 24][s * 24 + idx % 24] : 0.0;
        m = max(m, exp_of(v[i], idx < 288 ? __ldg(rx + idx / 24) : 0));
      }
      atomicMax(&s_em[which][s], m);
    }
    __syncthreads();
    if (s < nvalid) {
      m = s_em[which][s];
#pragma unroll
      for (int i = 0; i < kVals; ++i) {
        int const idx = i0 + i * kPer;
        if (idx < 288) {
          ll const x = to_fixed<4>(v[i], __ldg(rx + idx / 24), m);  // |x| <= 2^57
          int const hi = (int)((x + (1ll << 28)) >> 29), lo = (int)(x - ((ll)hi << 29));
          *reinterpret_cast<int2*>(&rows[idx / 24][s * 24 + idx % 24]) = make_int2(hi, lo);
        }
      }
    }
  }
  __syncthreads();
  int const p = t / 12, q = t % 12;
  bool const active = t < 144;
#pragma unroll 1
  for (int s = 0; s < kTS; ++s) {
    ll X[4][2];
    ull o = 0;
    if (active) {
      const int4* S = reinterpret_cast<const int4*>(&stage[q][s * 24]);
      const int4* Y = reinterpret_cast<const int4*>(&stage[12 + p][s * 24]);
      // O[s1][s2] = sum_c Y[s1][c] conj(S[s2][c]): al = O02 - O31, be = O13 - O20,
      // ev = O03 + O21, od = O12 + O30; D_0 = al + be, D_3 = i (be - al),
      // D_1 = -i (ev + od), D_2 = ev - od. Each sum as hi.hi and hi.lo + lo.hi.
      ll h[8], m[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) h[i] = m[i] = 0;
      // (ah, al), (bh, bl): limbs
      auto mac = [&](int i, int ah, int al, int bh, int bl) {
        h[i] += (ll)ah * bh;
        m[i] += (ll)ah * bl;
        m[i] += (ll)al * bh;
      };
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        int4 const y0 = Y[c], y1 = Y[3 + c], y2 = Y[6 + c], y3 = Y[9 + c];
        {
          int4 const x2 = S[6 + c];
          mac(0, y0.x, y0.y, x2.x, x2.y); mac(0, y0.z, y0.w, x2.z, x2.w);
          mac(1, y0.z, y0.w, x2.x, x2.y); mac(1, -y0.x, -y0.y, x2.z, x2.w);
          mac(6, y1.x, y1.y, x2.x, x2.y); mac(6, y1.z, y1.w, x2.z, x2.w);
          mac(7, y1.z, y1.w, x2.x, x2.y); mac(7, -y1.x, -y1.y, x2.z, x2.w);
        }
        {
          int4 const x3 = S[9 + c];
          mac(2, y1.x, y1.y, x3.x, x3.y); mac(2, y1.z, y1.w, x3.z, x3.w);
          mac(3, y1.z, y1.w, x3.x, x3.y); mac(3, -y1.x, -y1.y, x3.z, x3.w);
          mac(4, y0.x, y0.y, x3.x, x3.y); mac(4, y0.z, y0.w, x3.z, x3.w);
          mac(5, y0.z, y0.w, x3.x, x3.y); mac(5, -y0.x, -y0.y, x3.z, x3.w);
        }
        {
          int4 const x1 = S[3 + c];
          mac(0, -y3.x, -y3.y, x1.x, x1.y); mac(0, -y3.z, -y3.w, x1.z, x1.w);
          mac(1, -y3.z, -y3.w, x1.x, x1.y); mac(1, y3.x, y3.y, x1.z, x1.w);
          mac(4, y2.x, y2.y, x1.x, x1.y); mac(4, y2.z, y2.w, x1.z, x1.w);
          mac(5, y2.z, y2.w, x1.x, x1.y); mac(5, -y2.x, -y2.y, x1.z, x1.w);
        }
        {
          int4 const x0 = S[c];
          mac(2, -y2.x, -y2.y, x0.x, x0.y); mac(2, -y2.z, -y2.w, x0.z, x0.w);
          mac(3, -y2.z, -y2.w, x0.x, x0.y); mac(3, y2.x, y2.y, x0.z, x0.w);
          mac(6, y3.x, y3.y, x0.x, x0.y); mac(6, y3.z, y3.w, x0.z, x0.w);
          mac(7, y3.z, y3.w, x0.x, x0.y); mac(7, -y3.x, -y3.y, x0.z, x0.w);
        }
      }
      // in units of 2^58 input units
#pragma unroll
      for (int i = 0; i < 8; ++i) h[i] += (m[i] + (1ll << 28)) >> 29;
      X[0][0] = h[0] + h[2];  X[0][1] = h[1] + h[3];
      X[3][0] = h[1] - h[3];  X[3][1] = h[2] - h[0];
      X[1][0] = h[5] + h[7];  X[1][1] = -(h[4] + h[6]);
      X[2][0] = h[4] - h[6];  X[2][1] = h[5] - h[7];
#pragma unroll
      for (int i = 0; i < 8; ++i) o |= (ull)(X[i >> 1][i & 1] ^ (X[i >> 1][i & 1] >> 63));
    }
    // the position of the site's largest |D|'s top bit
    uint32_t const oh = __reduce_or_sync(0xffffffffu, (uint32_t)(o >> 32));
    uint32_t const ol = __reduce_or_sync(0xffffffffu, (uint32_t)o);
    if ((t & 31) == 0) {
      s_or[s & 1][t >> 5][0] = oh;
      s_or[s & 1][t >> 5][1] = ol;
    }
    __syncthreads();
    uint32_t ah = 0, al = 0;
#pragma unroll
    for (int w = 0; w < 5; ++w) {
      ah |= s_or[s & 1][w][0];
      al |= s_or[s & 1][w][1];
    }
    int const sh = 64 - __clzll((ll)(((ull)ah << 32) | al)) - 56;  // to |D| <= 2^56
    if (active && s < nvalid) {
      int const l = l0 + s;
      uint4* out = words + ((size_t)(l / kSites) * nf + fl) * kTileWords + ((size_t)(t >> 2) * kRows + l % kSites) * 4 + (t & 3);
#pragma unroll
      for (int mu = 0; mu < 4; ++mu) {
        uint32_t lo[2], hi[2];  // fields 0-3, 4-7
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          ll const v = X[mu][e];
          // to nearest even
          ull const d = (ull)(sh > 0 ? (v + (1ll << (sh - 1)) - 1 + ((v >> sh) & 1)) >> sh : v << -sh) + kBias;
          lo[e] = (uint32_t)d;  // bits 28-31: masked below
          hi[e] = (uint32_t)(d >> 28);
        }
        out[mu * kSites * 4] = make_uint4(__byte_perm(hi[0] >> 14, hi[1] >> 14, 0x5410), __byte_perm(hi[0], hi[1], 0x5410) & 0x3FFF3FFFu,
                                          __byte_perm(lo[0] >> 14, lo[1] >> 14, 0x5410) & 0x3FFF3FFFu,
                                          __byte_perm(lo[0], lo[1], 0x5410) & 0x3FFF3FFFu);
      }
      if (t == 0) {
        int const a = s_em[0][s], b = s_em[1][s];
        esc[fl * kMaxSites + l] = a == kNoScale || b == kNoScale ? kNoScale : a + b - 2100 + sh;
      }
    }
  }
}

// ---- the coefficients of the closed-form weight ------------------------------------
// coef[tile][mu][n / 2][32 sites][2] of the batch's sites. A lane is a site and a warp
// takes (mu, nu) and two lam at a time: which of an entry's terms vanish is then known
// at compile time, and E3(k, lam, nu, mu) of the six k serves the ten columns j of
// (mu, nu, lam).
struct CoefSmem {
  double tab[3][kQedTab][kSites];         // the tensor's factors per evaluation and site
  double zh[4][kSites];
  double w[3][HLBL_QED_NW][kSites];       // the weight functions
};
// kerv[K][A][B][C] of the lane's site, (R, S) the K-th pair; qed_tab_value's factors.
// The indices are compile-time constants: an entry has 0 to 4 terms, and what it has
// not costs no FP64 instruction (a vanishing term skipped at run time still did,
// predicated: the coefficients took 6.4 k per site, with the weights' quadrature it is
// 7.2 k now).
constexpr bool pair_is(int x, int y, int K) {
  int const r = comb_rho(K), s = comb_sigma(K);
  return (x == r && y == s) || (x == s && y == r);
}
template <int K, int A, int B, int C>
struct Entry {
  static constexpr int R = comb_rho(K), S = comb_sigma(K);
  static constexpr bool t0 = pair_is(A, B, K), t1 = pair_is(A, C, K), t2 = pair_is(B, C, K), f3 = A == B,
                        f4 = A == R || A == S, f5 = C == R || C == S;
  static constexpr bool none = !(t0 || t1 || t2 || f3 || f4 || f5);
  static __device__ __forceinline__ double get(const double (*tab)[kSites], int lane) {
    double v = 0.0;
    if constexpr (t0) v = A == S ? -tab[C][lane] : tab[C][lane];
    if constexpr (t1) {
      double const x = A == S ? -tab[4 + B][lane] : tab[4 + B][lane];
      v = t0 ? v + x : x;
    }
    if constexpr (t2) {
      double const x = B == S ? -tab[8 + A][lane] : tab[8 + A][lane];
      v = t0 || t1 ? v + x : x;
    }
    if constexpr (f3) {
      double const x = tab[12 + K][lane], w = tab[18 + C][lane];
      v = t0 || t1 || t2 ? fma(x, w, v) : x * w;
    }
    if constexpr (f4) {
      double const x = A == S ? tab[22 + R][lane] : -tab[22 + S][lane], w = tab[26 + 4 * B + C][lane];
      v = t0 || t1 || t2 || f3 ? fma(x, w, v) : x * w;
    }
    if constexpr (f5) {
      double const x = C == S ? tab[42 + R][lane] : -tab[42 + S][lane], w = tab[46 + 4 * A + B][lane];
      v = t0 || t1 || t2 || f3 || f4 ? fma(x, w, v) : x * w;
    }
    return v;
  }
};
// The ten columns j of (MU, NU, LAM): c[0..5] = E1 + E2 - E3, c[6 + tau] = sum_k E3(k)
// (zh_rho_k [sigma_k = tau] - zh_sigma_k [rho_k = tau])
template <int K, int MU, int NU, int LAM>
__device__ __forceinline__ void coef_k(const CoefSmem& sm, int lane, const double zh[4], double c[10]) {
  using E1 = Entry<K, MU, NU, LAM>;
  using E2 = Entry<K, NU, MU, LAM>;
  using E3 = Entry<K, LAM, NU, MU>;
  constexpr int R = comb_rho(K), S = comb_sigma(K);
  double v = 0.0;
  if constexpr (!E1::none) v = E1::get(sm.tab[0], lane);
  if constexpr (!E2::none) {
    double const e = E2::get(sm.tab[1], lane);
    v = E1::none ? e : v + e;
  }
  if constexpr (!E3::none) {
    double const e = E3::get(sm.tab[2], lane);
    v = E1::none && E2::none ? -e : v - e;
    c[6 + S] = fma(zh[R], e, c[6 + S]);
    c[6 + R] = fma(-zh[S], e, c[6 + R]);
  }
  c[K] = v;
}
template <int T>
__device__ __forceinline__ void coef_task(const CoefSmem& sm, int lane, const double zh[4], double2* __restrict__ out) {
  constexpr int MU = T >> 3, NU = (T >> 1) & 3, LAM = 2 * (T & 1);
  double c[2][10];
#pragma unroll
  for (int l = 0; l < 2; ++l)
#pragma unroll
    for (int j = 6; j < 10; ++j) c[l][j] = 0.0;
#define HG_COEF_K(K) coef_k<K, MU, NU, LAM>(sm, lane, zh, c[0]); coef_k<K, MU, NU, LAM + 1>(sm, lane, zh, c[1]);
  HG_COEF_K(0) HG_COEF_K(1) HG_COEF_K(2) HG_COEF_K(3) HG_COEF_K(4) HG_COEF_K(5)
#undef HG_COEF_K
#pragma unroll
  for (int j = 0; j < 10; ++j)
    out[(size_t)(MU * (kBtN / 2) + 8 * j + 2 * NU + (LAM >> 1)) * kSites] = make_double2(c[0][j], c[1][j]);
}
__device__ __forceinline__ void coef_cta(CoefSmem& sm, const WArgs& wa, const QedF32& qf, const Geometry& geo,
                                         const double* __restrict__ w, int block, ll s_begin, double* __restrict__ coef) {
  constexpr int kWarps = kDThreads / 32;
  int const t = threadIdx.x, lane = t & 31, warp = t >> 5;
  double const xu = wa.xunit;
  const PairBatch& batch = wa.batch;
  int const gsx[4] = {batch.p[0].gsx[0], batch.p[0].gsx[1], batch.p[0].gsx[2], batch.p[0].gsx[3]};
  int const yv[4] = {batch.p[0].yv[0], batch.p[0].yv[1], batch.p[0].yv[2], batch.p[0].yv[3]};
  ll const site = min(s_begin + (ll)kSites * block + lane, geo.V - 1);
  // e = 0: K(x, y), 1: K(y, x), 2: K(x, x - y)
  if (warp < 3) {
    double ww[HLBL_QED_NW];
    if (w == nullptr) {
      double a[4], b[4], X, c, Y;
      qed_args(geo, gsx, yv, xu, site, warp, a, b);
      hlbl_qed_invariants(a, b, &X, &c, &Y);
      qed_weights_fp64(wa.qp, qf, X, c, Y, ww);
    } else {
#pragma unroll
      for (int j = 0; j < HLBL_QED_NW; ++j) ww[j] = w[(size_t)(site * 3 + warp) * HLBL_QED_NW + j];
    }
#pragma unroll
    for (int j = 0; j < HLBL_QED_NW; ++j) sm.w[warp][j][lane] = ww[j];
  }
  __syncthreads();
  {
    int rel[4];
    rel_coords_fast(geo, gsx, site, rel);
    double xm[4], ym[4], xy[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      xm[r] = coord_map(rel[r], geo.global[r]) * xu;
      ym[r] = coord_map(mod_pos(yv[r], geo.global[r]), geo.global[r]) * xu;
      xy[r] = coord_map_diff(rel[r], yv[r], geo.global[r]) * xu;
      if (warp == 0) sm.zh[r][lane] = (double)coord_map_zerohalf(rel[r], geo.global[r]);
    }
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      double wv[HLBL_QED_NW];
#pragma unroll
      for (int j = 0; j < HLBL_QED_NW; ++j) wv[j] = sm.w[e][j][lane];
      const double* A = e == 1 ? ym : xm;
      const double* B = e == 0 ? ym : (e == 1 ? xm : xy);
#pragma unroll
      for (int i = 0; i < kQedTab; ++i)
        if (i % kWarps == warp) sm.tab[e][i][lane] = qed_tab_value(i, A, B, wv);
    }
  }
  __syncthreads();
  double zh[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) zh[r] = sm.zh[r][lane];
  double2* const out = reinterpret_cast<double2*>(coef) + (size_t)block * (kCoefPerSite / 2) * kSites + lane;
  if (warp == 4) return;  // four warps, one per scheduler
#pragma unroll 1
  for (int task = warp; task < 32; task += 4) {
    switch (task) {
#define HG_COEF_T(T) case T: coef_task<T>(sm, lane, zh, out); break;
#define HG_COEF_T4(T) HG_COEF_T(T) HG_COEF_T(T + 1) HG_COEF_T(T + 2) HG_COEF_T(T + 3)
      HG_COEF_T4(0) HG_COEF_T4(4) HG_COEF_T4(8) HG_COEF_T4(12)
      HG_COEF_T4(16) HG_COEF_T4(20) HG_COEF_T4(24) HG_COEF_T4(28)
#undef HG_COEF_T4
#undef HG_COEF_T
    }
  }
}

// One launch for both, so that the coefficients (FP64 pipe; first, as they take
// longest) and D formation (integer pipe) share the SMs. ncoef: 0 where the caller
// has coefficients; w: weights, or null to evaluate them here (exact mode). A
// weights kernel and one kernel for each took 98 + 118 + 170 us per 8,192 sites,
// this 282, and 230 with the vanishing terms left out at compile time.
__global__ void __launch_bounds__(kDThreads, 4)
site_kernel(const double* __restrict__ y, WArgs wa, QedF32 qf, Geometry geo, int f0, int nf, ll s_begin, int ncoef,
            const int* __restrict__ rowexp, const double* __restrict__ w, uint4* __restrict__ words, int* __restrict__ esc,
            double* __restrict__ coef, int* __restrict__ err) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  if (blockIdx.x < ncoef) {
    coef_cta(*reinterpret_cast<CoefSmem*>(smem_raw), wa, qf, geo, w, blockIdx.x, s_begin, coef);
    return;
  }
  int const d = blockIdx.x - ncoef;
  dform_cta(*reinterpret_cast<DSmem*>(smem_raw), y, wa.batch.p[0].src, geo, f0, d % nf, nf, d / nf, s_begin, rowexp, words,
            esc, err);
}
constexpr size_t kSiteSmem = sizeof(CoefSmem) > sizeof(DSmem) ? sizeof(CoefSmem) : sizeof(DSmem);

// ---- the products ------------------------------------------------------------------
constexpr int kStages = 3;
constexpr int kAPlane = kRows * 16 * 2;           // bytes of one digit of a chunk's A
constexpr int kBMax = part_chunk(0);              // bytes of a chunk's Bt digits
constexpr int kUnpackWarps = 16, kEWarps = 8, kWarpE0 = kUnpackWarps, kWarpMma = kWarpE0 + kEWarps, kWarpB = kWarpMma + 1;
constexpr int kThreads = 32 * (kWarpB + 1);
constexpr int kTmemCols = 512;
static_assert(kAcc * part_n(0) == kTmemCols, "eight accumulators of 64 columns");

struct __align__(1024) Smem {
  unsigned char A[kStages][kDig * kAPlane];
  unsigned char B[kStages][kBMax];
  ll F[64][kRows];                                // the tile's F as integers (each thread its own)
  uint64_t a_full[kStages], b_full[kStages], empty[kStages], acc_full, acc_free, mma_done;
  double red[kEWarps][2][2];
  int corr[2][kBtN];
  int col_sh[2][kBtN];                            // a column's exponent relative to the largest, as a high word
  int em_max[2];
  uint32_t taddr;
  int fail;
};
static_assert(sizeof(Smem) <= 232448, "shared memory above the 227 KB a CTA may have");

// instruction descriptor: D F32, A and B FP16, both K-major, M = 128
__device__ __forceinline__ uint32_t idesc(int n) {
  return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24);
}
__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t desc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d),
      "l"(a), "l"(b), "r"(desc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void tmem_ld4(uint32_t addr, uint32_t r[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
// kOff + digit, of two values -> the digits in FP16 (1024 + u is exact there)
template <uint32_t kOff>
__device__ __forceinline__ uint32_t dig2(uint32_t u) {
  uint32_t const x = u | 0x64006400u, k = 0x64006400u + kOff * 0x10001u;  // 1024 + u, 1024 + kOff
  __half2 const h = __hsub2(*reinterpret_cast<const __half2*>(&x), *reinterpret_cast<const __half2*>(&k));
  return *reinterpret_cast<const uint32_t*>(&h);
}

// a converged warp's wait: the same answer in every lane
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, volatile int* fail) {
  return __all_sync(0xffffffffu, tc::wait_or_fail(bar, parity, fail));
}

// Units (tile, flavour, part) over the CTAs. state[cta][fl]: the compensated sum
// over the batches; the last batch's launch writes partials.
template <int NF>
__global__ void __launch_bounds__(kThreads, 1)
digit_mma_kernel(const uint4* __restrict__ words, const int* __restrict__ esc, const unsigned char* __restrict__ bt,
                 const int* __restrict__ bem, const int* __restrict__ corr, const double* __restrict__ coef, int coef_tiled, int nsites, int first, int last,
                 double* __restrict__ state, double* __restrict__ partials, int* __restrict__ err) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
  int const t = threadIdx.x, warp = t >> 5, lane = t & 31;
  volatile int* const fail = &sm.fail;
  if (t == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&sm.a_full[i], 8);
      mbar_init(&sm.b_full[i], 1);
      mbar_init(&sm.empty[i], 1);
    }
    mbar_init(&sm.acc_full, 1);
    mbar_init(&sm.acc_free, kEWarps);
    mbar_init(&sm.mma_done, 1);
    fence_mbar_init();
    sm.fail = 0;
  }
  if (t < NF) {
    int m = kZeroExp;
    for (int n = 0; n < kBtN; ++n) m = max(m, bem[t * kBtN + n]);
    sm.em_max[t] = m;
  }
  if (warp == kWarpMma) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.taddr)),
                 "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  if (t < NF * kBtN) {
    int const m = sm.em_max[t / kBtN];
    sm.col_sh[t / kBtN][t % kBtN] = max(bem[t] - m, -900) * (1 << 20);
    sm.corr[t / kBtN][t % kBtN] = corr[t];
  }
  __syncthreads();
  uint32_t const tmem = sm.taddr;
  int const nunits = (nsites + kSites - 1) / kSites * NF * kParts;

  if (warp < kUnpackWarps) {
    // ---- A's digits: thread = (row, k / 8) of every other chunk ----------------------
    int const row = t & (kRows - 1), kc = (t >> 7) & 1, grp = t >> 8;
    int st = grp % kStages;
    uint32_t ph = 1;
    bool ok = true;
#pragma unroll 1
    for (int u = blockIdx.x; u < nunits && ok; u += gridDim.x) {
      const uint4* w4 = words + (size_t)(u / kParts) * kTileWords + ((size_t)(2 * grp + kc) * kRows + row) * 4;
      uint4 nx[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) nx[i] = __ldg(w4 + i);
#pragma unroll 1
      for (int c = grp; c < kChunks; c += 2) {
        uint4 cur[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) cur[i] = nx[i];
        if (c + 2 < kChunks) {
          w4 += 4 * kRows * 4;  // a chunk: 2 x 128 x 4 words
#pragma unroll
          for (int i = 0; i < 4; ++i) nx[i] = __ldg(w4 + i);
        }
        if (!warp_wait(&sm.empty[st], ph, fail)) { ok = false; break; }
        unsigned char* A = sm.A[st] + ((size_t)kc * kRows + row) * 16;
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          uint32_t d[2][4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            uint32_t const x = w == 0 ? cur[i].x : (w == 1 ? cur[i].y : (w == 2 ? cur[i].z : cur[i].w));
            d[1][i] = dig2<64>(x & 0x007F007Fu);
            d[0][i] = w == 0 ? dig2<128>((x >> 7) & 0x01FF01FFu) : dig2<64>((x >> 7) & 0x007F007Fu);
          }
#pragma unroll
          for (int e = 0; e < 2; ++e)
            *reinterpret_cast<uint4*>(A + (2 * w + e) * kAPlane) = make_uint4(d[e][0], d[e][1], d[e][2], d[e][3]);
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&sm.a_full[st]);
        // two chunks on
        if ((st += 2) >= kStages) { st -= kStages; ph ^= 1u; }
      }
    }
  } else if (warp == kWarpB) {
    // ---- Bt's digits -----------------------------------------------------------------
    if (lane == 0) {
      int st = 0, issued = 0;
      uint32_t ph = 1;
      bool ok = true;
#pragma unroll 1
      for (int u = blockIdx.x; u < nunits && ok; u += gridDim.x) {
        int const part = u % kParts, fl = (u / kParts) % NF, bytes = part_chunk(part);
        const unsigned char* b = bt + (size_t)fl * kBtBytes + part_base(part);
#pragma unroll 1
        for (int c = 0; c < kChunks; ++c) {
          if (!tc::wait_or_fail(&sm.empty[st], ph, fail)) { ok = false; break; }
          mbar_arrive_expect_tx(&sm.b_full[st], (uint32_t)bytes);
          bulk_g2s(sm.B[st], b + (size_t)c * bytes, (uint32_t)bytes, &sm.b_full[st]);
          ++issued;
          if (++st == kStages) { st = 0; ph ^= 1u; }
        }
      }
      // every copy lands before the CTA exits
      for (int i = max(0, issued - kStages); i < issued; ++i) mbar_wait(&sm.b_full[i % kStages], (uint32_t)(i / kStages) & 1u);
    }
  } else if (warp == kWarpMma) {
    // ---- MMA issue ---------------------------------------------------------------------
    int st = 0, nu = 0;
    uint32_t ph = 0;
    bool ok = true;
#pragma unroll 1
    for (int u = blockIdx.x; u < nunits && ok; u += gridDim.x, ++nu) {
      int const np = part_n(u % kParts);
      if (!warp_wait(&sm.acc_free, (uint32_t)(nu & 1) ^ 1u, fail)) break;
#pragma unroll 1
      for (int c = 0; c < kChunks; ++c) {
        if (!warp_wait(&sm.a_full[st], ph, fail) || !warp_wait(&sm.b_full[st], ph, fail)) { ok = false; break; }
        tc::tc_fence_after();
        uint64_t const a = tc::sdesc(smem_u32(sm.A[st]), kRows * 16, 128);
        uint64_t const b = tc::sdesc(smem_u32(sm.B[st]), kDig * np * 16, 128);
        if (tc::elect_one()) {
          // digit i of A with the digits j <= 7 - i of Bt, rows j np + n of one
          // operand, into the accumulators' columns (i + j) np + n: 12 products of up
          // to 256 columns (36 of 64 read A's digits from shared memory three times as
          // often, which took twice the time of the products)
#pragma unroll
          for (int i = 0; i < kDig; ++i)
#pragma unroll
            for (int r0 = 0; r0 < 64 * (kDig - i); r0 += 256) {
              int const rows = min(np * (kDig - i) - r0, 256);
              if (rows > 0)
                mma_f16(tmem + i * np + r0, a + (uint64_t)(i * (kAPlane >> 4)), b + (uint64_t)r0, idesc(rows),
                        i > 0 || c > 0 ? 1u : 0u);
            }
          tc::mma_commit(&sm.empty[st]);
          if (c == kChunks - 1) tc::mma_commit(&sm.acc_full);
        }
        __syncwarp();
        if (++st == kStages) { st = 0; ph ^= 1u; }
      }
    }
    // no product in flight when the CTA exits
    if (tc::elect_one()) {
      tc::mma_commit(&sm.mma_done);
      mbar_wait(&sm.mma_done, 0);
    }
    __syncwarp();
  } else {
    // ---- F from the accumulators, the dot ------------------------------------------------
    int const ew = warp - kWarpE0, mu = ew & 3, half = ew >> 2, row = mu * 32 + lane;
    uint32_t const lane_addr = tmem + ((uint32_t)(mu * 32) << 16);
    Neu run[NF];
    int nu = 0;
#pragma unroll 1
    for (int u = blockIdx.x; u < nunits; u += gridDim.x, ++nu) {
      int const part = u % kParts, fl = (u / kParts) % NF, site = u / (kParts * NF) * kSites + lane;
      int const nh = part_n(part) / 2, n0 = half * nh;
      if (!warp_wait(&sm.acc_full, (uint32_t)nu & 1u, fail)) break;
      tc::tc_fence_after();
#pragma unroll 1
      for (int n = n0; n < n0 + nh; n += 4) {
        uint32_t r[kAcc][4];
#pragma unroll
        for (int d = 0; d < kAcc; ++d) tmem_ld4(lane_addr + d * 2 * nh + n, r[d]);
        tc::tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          int x[kAcc];
#pragma unroll
          for (int d = 0; d < kAcc; ++d) x[d] = __float2int_rn(__uint_as_float(r[d][i]));
          ll const hi = ((((((ll)x[0] << 7) + x[1]) << 7) + x[2]) << 7) + x[3];
          ll const lo = ((((((ll)x[4] << 7) + x[5]) << 7) + x[6]) << 7) + x[7] + sm.corr[fl][part_n0(part) + n + i];
          sm.F[n + i][row] = (hi << 19) + ((lo + 256) >> 9);  // F 2^-58, below 2^63
        }
      }
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&sm.acc_free);
      double part_sum = 0.0;
      if (site < nsites) {
        // two columns at cf + step n / 2
        int const nc = mu * kBtN + part_n0(part), step = coef_tiled ? kSites : 1;
        const double2* cf = reinterpret_cast<const double2*>(coef) +
                            (coef_tiled ? ((size_t)(site / kSites) * (kCoefPerSite / 2) + nc / 2) * kSites + lane
                                        : ((size_t)site * kCoefPerSite + nc) / 2);
        const int* shp = &sm.col_sh[fl][part_n0(part)];
#pragma unroll 4
        for (int n = n0; n < n0 + nh; n += 2) {
          double2 const c2 = __ldg(cf + (size_t)(n / 2) * step);
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            ll const v = sm.F[n + i][row];
            double const f = (double)v;
            // times the column's power of two
            double const g = __hiloint2double(__double2hiint(f) + (v != 0 ? shp[n + i] : 0), __double2loint(f));
            part_sum = fma(i == 0 ? c2.x : c2.y, g, part_sum);
          }
        }
        int const e = esc[fl * kMaxSites + site], m = sm.em_max[fl];
        part_sum = e == kNoScale || m == kNoScale ? __longlong_as_double(0x7FF8000000000000ll)
                                               : ldexp(part_sum, e + m - 1078 + 58);
      }
      if (NF == 1 || fl == 0) run[0].add(-part_sum);
      else run[NF - 1].add(-part_sum);
    }
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      Neu v = run[f];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        double const os = __shfl_down_sync(0xffffffffu, v.s, o);
        double const oc = __shfl_down_sync(0xffffffffu, v.c, o);
        v.add(os);
        v.c += oc;
      }
      if (lane == 0) { sm.red[ew][f][0] = v.s; sm.red[ew][f][1] = v.c; }
    }
  }
  __syncthreads();
  if (t < NF && !*fail) {
    Neu s;
    double* const mine = state + ((size_t)blockIdx.x * 2 + t) * 2;
    if (!first) { s.s = mine[0]; s.c = mine[1]; }
    for (int w = 0; w < kEWarps; ++w) { s.add(sm.red[w][t][0]); s.c += sm.red[w][t][1]; }
    mine[0] = s.s;
    mine[1] = s.c;
    if (last) partials[(size_t)blockIdx.x * NF + t] = s.get();
  }
  if (t == 0 && *fail && err) atomicExch(err, kErrWaitTimeout);
  if (warp == kWarpMma)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
}

// ---- the work buffer ------------------------------------------------------------------
struct Ws {
  size_t words, bt, coef, state, esc, bem, rowexp, corr, total;  // byte offsets
};
static int ws_tiles(ll V) { return (int)std::min<ll>(kMaxTiles, (V + kSites - 1) / kSites); }
static Ws ws_layout(ll V, int nsm) {
  Ws w{};
  size_t o = 0;
  auto take = [&](size_t bytes) {
    size_t const at = o;
    o += (bytes + 255) / 256 * 256;
    return at;
  };
  size_t const tiles = (size_t)ws_tiles(V);
  w.words = take(tiles * 2 * kTileWords * sizeof(uint4));
  w.bt = take(2 * kBtBytes);
  w.coef = take(tiles * kSites * kCoefPerSite * sizeof(double));
  w.state = take((size_t)nsm * 4 * sizeof(double));
  w.esc = take(2 * kMaxSites * sizeof(int));
  w.bem = take(2 * kBtN * sizeof(int));
  w.rowexp = take(2 * kRowExp * sizeof(int));
  w.corr = take(2 * kBtN * sizeof(int));
  w.total = o;
  return w;
}

template <int NF>
static void launch_t(int nsm, cudaStream_t st, const double* y, const WArgs& wa, const QedF32& qf, const Geometry& geo,
                     const P2Args& a, const double* dz, const double* g_dzu, const double* g_dzsu, void* ws,
                     double* partials, int* err) {
  Ws const l = ws_layout(geo.V, nsm);
  unsigned char* const p = static_cast<unsigned char*>(ws);
  uint4* const words = reinterpret_cast<uint4*>(p + l.words);
  double* const coef = reinterpret_cast<double*>(p + l.coef);
  int* const esc = reinterpret_cast<int*>(p + l.esc);
  int* const bem = reinterpret_cast<int*>(p + l.bem);
  int* const corr = reinterpret_cast<int*>(p + l.corr);
  int* const rowexp = reinterpret_cast<int*>(p + l.rowexp);
  brow_kernel<<<NF, kRowThreads, 0, st>>>(dz, g_dzu, g_dzsu, rowexp);
  bdig_build_kernel<<<dim3(kBtN, NF), kBtK, 0, st>>>(dz, g_dzu, g_dzsu, rowexp, p + l.bt, bem, corr);
  for (ll s0 = 0; s0 < geo.V; s0 += kMaxSites) {
    int const n = (int)std::min<ll>(kMaxSites, geo.V - s0), cta = (n + kTS - 1) / kTS;
    const double* cf = static_cast<const double*>(a.coef);
    int const ncoef = cf != nullptr ? 0 : (n + kSites - 1) / kSites;
    site_kernel<<<cta * NF + ncoef, kDThreads, ncoef > 0 ? kSiteSmem : sizeof(DSmem), st>>>(
        y, wa, qf, geo, a.f0, NF, s0, ncoef, rowexp, a.w, words, esc, coef, err);
    cf = cf != nullptr ? cf + (size_t)s0 * kCoefPerSite : coef;
    digit_mma_kernel<NF><<<nsm, kThreads, sizeof(Smem), st>>>(words, esc, p + l.bt, bem, corr, cf, a.coef == nullptr, n, s0 == 0,
                                                              s0 + n >= geo.V, reinterpret_cast<double*>(p + l.state),
                                                              partials, err);
  }
}

}  // namespace dig

int p2dig_init() {
  cudaError_t e = cudaFuncSetAttribute(dig::site_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dig::kSiteSmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(dig::digit_mma_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(dig::Smem));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(dig::digit_mma_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(dig::Smem));
  return e == cudaSuccess ? HLBL_OK : cuda_fail(e, "digit product smem attribute");
}

size_t p2dig_ws_bytes(long long V, int nsm) { return dig::ws_layout(V, nsm).total; }

void p2dig_launch(int nf, int nsm, cudaStream_t st, const double* y, const WArgs& wa, const QedF32& qf, const Geometry& geo,
                  const P2Args& a, const double* dz, const double* g_dzu, const double* g_dzsu, void* ws,
                  double* partials, int* err) {
  if (nf == 2) dig::launch_t<2>(nsm, st, y, wa, qf, geo, a, dz, g_dzu, g_dzsu, ws, partials, err);
  else dig::launch_t<1>(nsm, st, y, wa, qf, geo, a, dz, g_dzu, g_dzsu, ws, partials, err);
}

}  // namespace hg
