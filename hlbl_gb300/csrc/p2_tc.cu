// p2_tc.cu -- pass 2 of the mixed-precision path on the 5th-generation tensor
// cores (tcgen05), the same sum as p2_kernel<float, 2, TS>:
//   F[mu][n] = sum_k Dr_mu[k] Bt[k][n],  dtmp = -sum_{mu,n} coef[mu][n] F[mu][n]
// (ker_4pt_contraction, cuda_lattice.cu:277-484, restructured as in
// contract_kernels.cuh).
//
// Per CTA (one per SM, persistent; tiles of 32 sites of all pairs from a common
// queue) and per phase (tile, flavour f): the 128 x 160 product F = A . B^T, A = Dr with rows
// (mu, site) = mu*32 + site and K = 288 = (p, q, re/im), B = Bt^T. Products
// are FP32 in the 3xTF32 form A_hi B_hi + A_hi B_lo + A_lo B_hi (hi = the
// TF32 rounding, lo = the TF32 rounding of the rest), accumulated in TMEM.
//
// Warp roles (19 warps):
//   0      TMA producer of the FP32 input rows (S = x[1-f] rows q, Y = y[f]
//          rows p: 3 KB per (flavour, ia, tile)) -- one thread
//   1      TMA producer of the B chunks (16 k x 160 n, hi and lo, 20 KB) -- one thread
//   3      TMEM allocation; tcgen05.mma issue and commits
//   2, 4-14  D formation, three groups of four warps on every third chunk of
//          16 k (8 (p, q): half of a block of 4 p x 4 q): warp j of a group
//          forms the chunk's j-th pair of (p, q) (one Y row, two S rows) for
//          its lane's site: O = Y conj(S) spin blocks -> D_mu -> hi/lo ->
//          shared memory in the K-major no-swizzle core-matrix layout
//   15-18  epilogue: one TMEM lane quadrant each (warp % 4 = mu); per phase,
//          the F rows from TMEM dotted with the QED coefficients of the
//          row's site; the quadrant's sum is stored per (tile, flavour), and
//          the tiles' sums are added in a fixed order afterwards, whichever
//          CTA took them
// The tensor cores accumulate in FP32 with truncation (biased toward zero),
// so the error grows with the number of MMAs added into one accumulator and
// the small hi.lo and lo.hi products lose most of their bits if added into
// the large hi.hi sum. Three accumulators of 160 TMEM columns: the
// corrections go to their own, and the hi.hi sum of chunks 0-8 and of
// chunks 9-17 to the two main buffers; the epilogue adds the second half
// and the corrections into the first (FP32, round-to-nearest) before the
// dot. The two main buffers swap roles every phase: the next phase's first
// half only waits for that fold, its second half for the dot.
// Pipelines (mbarriers; every wait bounded, kWaitLimit polls):
//   rows -> D warps (S rows of a block in a ring of 2 blocks, Y rows of a
//   p-block by halves in a ring of 3),
//   D warps and B producer -> MMA (operand stages, a ring of 5 or 6: one
//   barrier per stage, one commit per chunk frees it),
//   MMA -> epilogue (acc_full), epilogue -> MMA (folded, dotted).
//
// Inputs are the FP32 tile copies of the blocks (x32/y32: [f][ia][tile][2][6][16][4] floats, f32_tile_off: a site's
// 24 components as six 16-byte groups, 32 sites per tile in two halves), so
// pass 2 reads half the bytes of the FP64 blocks and converts nothing.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "contract_kernels.cuh"
#include "hlbl_gb300.h"
#include "hlbl_internal.h"
#include "p2_tc.h"
#include "tc_ops.cuh"

namespace hg {
namespace tc {

constexpr int kSites = 32;                 // sites per tile
constexpr int kM = 128;                    // MMA rows: (mu, site)
constexpr int kKc = 16;                    // K per chunk
constexpr int kChunks = kBtK / kKc;        // 18
// A and B rings of the same depth (OpT::kStages: 5 for TF32 operands, 10 for
// FP16), released by one commit per chunk: the tensor pipe's completion
// reaches the waiting producers about 2,500 cycles after a chunk is issued, so
// several chunks must be in flight to keep it busy; one commit per chunk frees
// the A and the B stage (a deeper ring for one of them with a second commit
// per chunk measured slower).
// K order: blocks of 4 p x 4 q (two chunks each), q-blocks inner, so both row
// sets stream through small rings instead of one being held for a whole
// phase: the S rows 4 bq..4 bq+3 of a block (a ring of two blocks; fetched
// again, from L2, for each p-block) and the Y rows of a p-block by halves,
// half h (rows 4 bp + 2h, 4 bp + 2h + 1) read by each D group in one of its
// three chunks (a ring of three halves). This leaves room for five A and B stages.
constexpr int kRowsPerGroup = 4, kBlocksQ = 3;
constexpr int kYRows = 2;
constexpr int kBlocks = 9;  // per phase: 3 p-blocks x 3 q-blocks
constexpr int kHalf = kChunks / 2;               // chunks per main-accumulator half
constexpr uint32_t kCorrCol = 2 * kBtN;          // the correction accumulator's first column
constexpr int kAPart = kM * kKc;           // floats per A part (hi or lo)
constexpr int kBPart = kBtN * kKc;         // floats per B part
// The MMA warp shares its scheduler (warp % 4) with the fewest others: of 19
// warps the fourth scheduler has four. D warps: 2 and 4-14.
constexpr int kWarpRows = 0, kWarpB = 1, kWarpMma = 3, kDWarps = 12;
constexpr int kDGroup = 4;  // D warps per chunk (a group); kDGroups chunks in flight
constexpr int kDGroups = kDWarps / kDGroup;
constexpr int kWarpE0 = 3 + kDWarps, kEWarps = 4;
constexpr int kThreads = 32 * (kWarpE0 + kEWarps);
// The CTAs take their units (pair, tile) from a common counter: at 663,552
// sites the same number of tiles each took 2.50 to 3.45 ms (both SMs of a TPC
// the same time, not the same TPCs from run to run), so that a fixed share each
// made the slowest hold the kernel. The row producer draws them, a few ahead,
// and hands them to the other warps through a small queue.
constexpr int kQueue = 4;
constexpr int kQueueReaders = 2 + kDWarps + kEWarps;  // B producer, MMA, D and epilogue warps
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kRowBytes = kRowF32 * 4;  // 3072

// Operand type of the products (both TF32 or both FP16; D is F32 either way).
// FP16: the same 3-term split as TF32 (hi = the rounding of the value, lo =
// the rounding of the rest: 11 + 11 significant bits) in half the bytes, with
// one MMA of K = 16 per product and chunk instead of two of K = 8, so the
// rings hold twice the chunks. FP16's exponent range is met by power-of-two
// scales: A by 2^(15 - e) with 2^e above the bound 24 max|Y| max|S| of every
// D value (from the per-flavour maxima the tile copies carry), B by the same
// rule from max|Bt| per pair and flavour; the epilogue divides each row's dot
// by the product (exact). The bytes saved go to deeper row rings (four S
// blocks, six Y halves instead of two and three), which the D warps were
// waiting on, and to seven operand stages.
template <bool F16> struct OpT;
// kSGroups, kYSlots: depths of the S-block and Y-half rings
// kBParts: B as hi + lo (TF32) or hi + lo + lo2 (FP16, split from the FP64
// value: ~33 significant bits, as B's rounding error would repeat at every
// site of a pair)
template <> struct OpT<false> {
  static constexpr int kStages = 5, kElem = 4, kSGroups = 2, kYSlots = 3, kBParts = 2;
  static constexpr uint32_t kFmt = 2;  // TF32
};
template <> struct OpT<true> {
  static constexpr int kStages = 6, kElem = 2, kSGroups = 4, kYSlots = 6, kBParts = 3;
  static constexpr uint32_t kFmt = 0;  // F16
};
// instruction descriptor: D F32, A and B of the operand type, both K-major,
// N = 160, M = 128
template <bool F16>
constexpr uint32_t idesc() {
  return (1u << 4) | (OpT<F16>::kFmt << 7) | (OpT<F16>::kFmt << 10) | ((uint32_t)(kBtN >> 3) << 17) |
         ((uint32_t)(kM >> 4) << 24);
}
constexpr uint32_t kIdesc = idesc<false>();

template <bool F16>
struct __align__(1024) SmemT {
  static constexpr int kSt = OpT<F16>::kStages;
  static constexpr int kAPartB = kAPart * OpT<F16>::kElem, kBPartB = kBPart * OpT<F16>::kElem;  // bytes
  static constexpr int kSGroups = OpT<F16>::kSGroups, kYSlots = OpT<F16>::kYSlots;
  float S[kSGroups][kRowsPerGroup][kRowF32];
  float Y[kYSlots][kYRows][kRowF32];
  __align__(16) unsigned char A[kSt][2][kAPartB];
  __align__(16) unsigned char B[kSt][OpT<F16>::kBParts][kBPartB];
  uint64_t s_full[kSGroups], s_empty[kSGroups], y_full[kYSlots], y_empty[kYSlots];
  uint64_t full[kSt], empty[kSt];  // operand stages: A by a D group, B by its copy
  uint64_t acc_full, folded, dotted, mma_done;
  uint64_t q_full[kQueue], q_empty[kQueue];
  uint32_t unit[kQueue];  // the queue of this CTA's (pair, tile) units
  uint32_t taddr;
  int fail, b_last;
};
using Smem = SmemT<false>;
static_assert(sizeof(SmemT<false>) <= 232448 && sizeof(SmemT<true>) <= 232448,
              "pass-2 shared memory above the 227 KB a CTA may have");

// FP16 hi and lo parts of two values, packed as the MMA reads them (the first
// value in the low half)
__device__ __forceinline__ void f16_split2(float a, float b, uint32_t& hi, uint32_t& lo) {
  __half2 const h = __floats2half2_rn(a, b);
  float2 const f = __half22float2(h);
  __half2 const l = __floats2half2_rn(a - f.x, b - f.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}
// 2^(15 - e), as far as FP32 has it
__host__ __device__ __forceinline__ float f16_scale_exp(int e) {
  int const k = 15 - e;
  return ldexpf(1.f, k < -126 ? -126 : (k > 127 ? 127 : k));
}
// 2^(15 - e) for the smallest e with bound < 2^e: scales values bounded by
// `bound` into FP16's range with a factor of two to spare (1 for bound 0)
__host__ __device__ __forceinline__ float f16_scale(float bound) {
  if (!(bound > 0.f) || !(bound <= 3.0e38f)) return 1.f;  // zero, NaN or infinite inputs
  int e;
  frexpf(bound, &e);  // bound = m 2^e, m in [0.5, 1)
  return f16_scale_exp(e);
}

__device__ __forceinline__ uint32_t tf32_rna(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}
// The same rounding (to nearest, ties away from zero, the low 13 bits
// cleared) on the integer pipe, for finite x: adding half a TF32 unit to the
// magnitude bits carries into the kept bits exactly when the dropped part is
// at least half; a carry into the exponent is the correct round-up. The
// D-formation warps round 16 values per (p, q) pair this way.
__device__ __forceinline__ float tf32_round(float x) {
  return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xFFFFE000u);
}
__device__ __forceinline__ void mma_tf32(uint32_t d, uint64_t a, uint64_t b, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}" ::"r"(d),
      "l"(a), "l"(b), "r"(kIdesc), "r"(acc));
}
// The four products of a chunk (hi.hi into d; hi.lo, lo.hi and hi.lo2 into dc)
// and the commit that frees its stage, issued by one elected lane of the
// converged warp: predicated instructions, no branch.
__device__ __forceinline__ void mma_chunk_f16(uint32_t d, uint32_t dc, uint64_t ahi, uint64_t alo, uint64_t bhi,
                                              uint64_t b_part, uint32_t acc_d, uint32_t acc_c, uint64_t* bar) {
  asm volatile(
      "{\n .reg .pred p, q, r, t;\n"
      " elect.sync _|p, 0xffffffff;\n"
      " setp.ne.b32 q, %7, 0;\n setp.ne.b32 r, %8, 0;\n setp.eq.b32 t, 0, 0;\n"
      " @p tcgen05.mma.cta_group::1.kind::f16 [%0], %2, %4, %9, q;\n"
      " @p tcgen05.mma.cta_group::1.kind::f16 [%1], %2, %5, %9, r;\n"
      " @p tcgen05.mma.cta_group::1.kind::f16 [%1], %3, %4, %9, t;\n"
      " @p tcgen05.mma.cta_group::1.kind::f16 [%1], %2, %6, %9, t;\n"
      " @p tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%10];\n}" ::"r"(d),
      "r"(dc), "l"(ahi), "l"(alo), "l"(bhi), "l"(bhi + b_part), "l"(bhi + 2 * b_part), "r"(acc_d), "r"(acc_c),
      "r"(idesc<true>()), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t addr, const float v[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(addr),
      "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])),
      "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])), "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])),
      "r"(__float_as_uint(v[8])), "r"(__float_as_uint(v[9])), "r"(__float_as_uint(v[10])), "r"(__float_as_uint(v[11])),
      "r"(__float_as_uint(v[12])), "r"(__float_as_uint(v[13])), "r"(__float_as_uint(v[14])), "r"(__float_as_uint(v[15]))
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ---- the QED-weighted dot of one row (mu = MU, fixed) ------------------------------
// The row's contribution is sum_n coef[MU][n] F[n] with n = (j, nu, lam),
// coef[MU][(k, nu, lam)] = E1(k, MU, nu, lam) + E2(k, nu, MU, lam) - E3(k, lam, nu, MU)
// (k < 6) and coef[MU][(6 + tau, nu, lam)] = sum_k c_k(tau) E3(k, lam, nu, MU)
// with c_k(tau) = [sigma_k = tau] zh_rho_k - [rho_k = tau] zh_sigma_k, where
// Ee(k, a, b, c) = kerv[k][a][b][c] of the stand-in tensor at the argument
// pair e: (xm, ym), (ym, xm), (xm, x - y) (hlbl_qed_entry: six terms w_0..w_5,
// each a Kronecker structure times coordinates). For fixed k the columns of
// F form a 4 x 4 matrix G[nu][lam], and each term's sum over (nu, lam)
// reduces to rows G.v, columns u.G, forms u.G.v, the trace and the
// antisymmetric part G[r][s] - G[s][r]; the sums below are those reductions.
struct SiteQ {
  float xm[4], ym[4], xmy[4], zh[4];
  float w[3][HLBL_QED_NW];
};

__device__ __forceinline__ float row_dot(const float* G, int i, const float* v) {
  return fmaf(G[4 * i + 3], v[3], fmaf(G[4 * i + 2], v[2], fmaf(G[4 * i + 1], v[1], G[4 * i] * v[0])));
}
__device__ __forceinline__ float col_dot(const float* G, int i, const float* u) {
  return fmaf(u[3], G[12 + i], fmaf(u[2], G[8 + i], fmaf(u[1], G[4 + i], u[0] * G[i])));
}

// sum_{nu,lam} E3(k, lam, nu, MU) G[nu][lam]; gx = G.xm, gz = G.xmy (rows),
// zg = xmy.G (columns), xGx = xm.G.xm, tr = trace(G)
template <int MU, int K>
__device__ __forceinline__ float d3(const float* G, const SiteQ& q, const float* gx, const float* gz,
                                    const float* zg, float xGx, float tr) {
  constexpr int r = comb_rho(K), s = comb_sigma(K);
  const float* x = q.xm;
  const float* y = q.xmy;
  const float* w = q.w[2];
  float const anti = G[4 * r + s] - G[4 * s + r];
  float v = -w[0] * x[MU] * anti;
  v = fmaf(w[3] * (x[r] * y[s] - x[s] * y[r]) * (x[MU] + y[MU]), tr, v);
  v = fmaf(w[4] * y[MU], x[r] * zg[s] - x[s] * zg[r], v);
  if constexpr (MU == s) v += w[1] * zg[r] + w[2] * (gx[r] - gz[r]) + w[5] * y[r] * xGx;
  if constexpr (MU == r) v -= w[1] * zg[s] + w[2] * (gx[s] - gz[s]) + w[5] * y[s] * xGx;
  return v;
}

// j = K < 6: E1 + E2 - E3 against G = F[(K, ., .)]
template <int MU, int K>
__device__ __forceinline__ float dot_k(const float* G, const SiteQ& q) {
  constexpr int r = comb_rho(K), s = comb_sigma(K);
  const float* xm = q.xm;
  const float* ym = q.ym;
  const float* xmy = q.xmy;
  float gx[4], gy[4], gz[4], zg[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    gx[i] = row_dot(G, i, xm);
    gy[i] = row_dot(G, i, ym);
  }
  gz[r] = row_dot(G, r, xmy); gz[s] = row_dot(G, s, xmy);
  zg[r] = col_dot(G, r, xmy); zg[s] = col_dot(G, s, xmy);
  float const ygr = col_dot(G, r, ym), ygs = col_dot(G, s, ym);  // ym.G
  float const xgr = col_dot(G, r, xm), xgs = col_dot(G, s, xm);  // xm.G
  float const yGy = fmaf(ym[3], gy[3], fmaf(ym[2], gy[2], fmaf(ym[1], gy[1], ym[0] * gy[0])));
  float const xGx = fmaf(xm[3], gx[3], fmaf(xm[2], gx[2], fmaf(xm[1], gx[1], xm[0] * gx[0])));
  float const tr = G[0] + G[5] + G[10] + G[15];
  float const anti = G[4 * r + s] - G[4 * s + r];
  const float* w1 = q.w[0];
  const float* w2 = q.w[1];
  // E1: (a, b, c) = (MU, nu, lam) at (xm, ym)
  float v = w1[2] * (xm[MU] - ym[MU]) * anti;
  v = fmaf(w1[3] * (xm[r] * ym[s] - xm[s] * ym[r]), gx[MU] + gy[MU], v);
  v = fmaf(w1[5] * xm[MU], ym[r] * xgs - ym[s] * xgr, v);
  if constexpr (MU == r) v += w1[0] * gx[s] + w1[1] * ygs - w1[4] * xm[s] * yGy;
  if constexpr (MU == s) v += -w1[0] * gx[r] - w1[1] * ygr + w1[4] * xm[r] * yGy;
  // E2: (a, b, c) = (nu, MU, lam) at (ym, xm)
  v = fmaf(w2[1] * xm[MU], anti, v);
  v = fmaf(w2[3] * (ym[r] * xm[s] - ym[s] * xm[r]), gy[MU] + gx[MU], v);
  v = fmaf(w2[4] * xm[MU], ym[r] * gx[s] - ym[s] * gx[r], v);
  v = fmaf(w2[5] * ym[MU], xm[r] * ygs - xm[s] * ygr, v);
  if constexpr (MU == s) v += w2[0] * gy[r] - w2[2] * (ygr - xgr);
  if constexpr (MU == r) v += -w2[0] * gy[s] + w2[2] * (ygs - xgs);
  // - E3: (a, b, c) = (lam, nu, MU) at (xm, x - y)
  return v - d3<MU, K>(G, q, gx, gz, zg, xGx, tr);
}

// j = 6 + TAU: sum_k c_k(TAU) E3(k, lam, nu, MU) against G = F[(6 + TAU, ., .)]
template <int MU, int TAU>
__device__ __forceinline__ float dot_zh(const float* G, const SiteQ& q) {
  float gx[4], gz[4], zg[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    gx[i] = row_dot(G, i, q.xm);
    gz[i] = row_dot(G, i, q.xmy);
    zg[i] = col_dot(G, i, q.xmy);
  }
  const float* xm = q.xm;
  float const xGx = fmaf(xm[3], gx[3], fmaf(xm[2], gx[2], fmaf(xm[1], gx[1], xm[0] * gx[0])));
  float const tr = G[0] + G[5] + G[10] + G[15];
  float v = 0.f;
  auto term = [&](auto kc) {
    constexpr int k = decltype(kc)::value;
    constexpr int r = comb_rho(k), g = comb_sigma(k);
    if constexpr (g == TAU || r == TAU) {
      float const e = d3<MU, k>(G, q, gx, gz, zg, xGx, tr);
      if constexpr (g == TAU) v = fmaf(q.zh[r], e, v);
      if constexpr (r == TAU) v = fmaf(-q.zh[g], e, v);
    }
  };
  term(std::integral_constant<int, 0>{});
  term(std::integral_constant<int, 1>{});
  term(std::integral_constant<int, 2>{});
  term(std::integral_constant<int, 3>{});
  term(std::integral_constant<int, 4>{});
  term(std::integral_constant<int, 5>{});
  return v;
}

// One phase's row: sum_n coef[MU][n] F[n], F at column c of this warp's lane
// quadrant (16 columns = one 4 x 4 matrix per j).
template <int MU>
__device__ __forceinline__ float epilogue_row(uint32_t lane_addr, uint32_t c, const SiteQ& q) {
  float f[16], a = 0.f;
#define HG_TC_K(J)                      \
  tmem_ld16(lane_addr + c + 16 * J, f); \
  tmem_wait_ld();                       \
  a += dot_k<MU, J>(f, q);
#define HG_TC_T(J)                      \
  tmem_ld16(lane_addr + c + 16 * J, f); \
  tmem_wait_ld();                       \
  a += dot_zh<MU, J - 6>(f, q);
  HG_TC_K(0) HG_TC_K(1) HG_TC_K(2) HG_TC_K(3) HG_TC_K(4) HG_TC_K(5)
  HG_TC_T(6) HG_TC_T(7) HG_TC_T(8) HG_TC_T(9)
#undef HG_TC_K
#undef HG_TC_T
  return a;
}

// Generic QED path: one phase's row dotted with the row's coefficients,
// read from the FP32 coefficient layout (crow: this row's (tile, mu, site)
// base; group g of four n at crow + g*128), one 16-column block of F per j.
// The next block's coefficients are loaded while the current one is dotted.
__device__ __forceinline__ float epilogue_row_generic(uint32_t lane_addr, uint32_t c, const float* crow) {
  float f[16], a = 0.f;
  float4 cf[4], cn[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) cf[i] = __ldg(reinterpret_cast<const float4*>(crow + i * 128));
#pragma unroll 1
  for (int jj = 0; jj < 10; ++jj) {
    if (jj + 1 < 10) {
#pragma unroll
      for (int i = 0; i < 4; ++i) cn[i] = __ldg(reinterpret_cast<const float4*>(crow + ((jj + 1) * 4 + i) * 128));
    }
    tmem_ld16(lane_addr + c + 16 * jj, f);
    tmem_wait_ld();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      a = fmaf(cf[i].x, f[4 * i], a);
      a = fmaf(cf[i].y, f[4 * i + 1], a);
      a = fmaf(cf[i].z, f[4 * i + 2], a);
      a = fmaf(cf[i].w, f[4 * i + 3], a);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) cf[i] = cn[i];
  }
  return a;
}

// The D formation's closed forms of D_mu from the spin-block products follow
// from these phases (i^((2 - g5g_ph(mu, s1)) & 3) for s1 = 0..3).
constexpr int d_ph(int mu, int s1) { return (6 - g5g_ph(mu, s1)) & 3; }
static_assert(d_ph(0, 0) == 0 && d_ph(0, 1) == 0 && d_ph(0, 2) == 2 && d_ph(0, 3) == 2, "D_0 = a0 + a1 - a2 - a3");
static_assert(d_ph(3, 0) == 3 && d_ph(3, 1) == 1 && d_ph(3, 2) == 3 && d_ph(3, 3) == 1, "D_3 = i (a1 + a3 - a0 - a2)");
static_assert(d_ph(1, 0) == 3 && d_ph(1, 1) == 3 && d_ph(1, 2) == 3 && d_ph(1, 3) == 3, "D_1 = -i (b0 + b1 + b2 + b3)");
static_assert(d_ph(2, 0) == 0 && d_ph(2, 1) == 2 && d_ph(2, 2) == 0 && d_ph(2, 3) == 2, "D_2 = b0 - b1 + b2 - b3");

// ---- the kernel ------------------------------------------------------------------
// kGeneric: the QED weighting from the coefficient tensor of args.coef (any
// QED kernel, qed_provider.cuh) instead of the stand-in's closed form.
// kF16: FP16 operands (OpT<true>); btu then holds FP16 parts and bscale the
// B scale per (pair, flavour).
template <bool kGeneric, bool kF16>
__global__ void __launch_bounds__(kThreads, 1)
p2tc_kernel(TcBatch tb, Geometry geo, P2Args args, const void* __restrict__ btu,
            const float* __restrict__ bscale, int npairs, double* __restrict__ tsum,
            unsigned* __restrict__ next_unit, int* __restrict__ err) {
  using Sm = SmemT<kF16>;
  constexpr int kSt = Sm::kSt, kSGroups = Sm::kSGroups, kYSlots = Sm::kYSlots;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  Sm& sm = *reinterpret_cast<Sm*>(smem_raw);
  volatile int* fail = &sm.fail;
  int const t = threadIdx.x, warp = t >> 5, lane = t & 31;
  uint32_t const ntiles = (uint32_t)((geo.V + kSites - 1) / kSites), nunits = ntiles * (uint32_t)npairs;
  const float* __restrict__ y32 = tb.y32;
  auto row_ptr = [&](const float* base, int f, int ia, uint32_t tile) {
    return base + ((size_t)(f * 12 + ia) * ntiles + tile) * kRowF32;
  };

  if (t == 0) {
    for (int i = 0; i < kSGroups; ++i) { mbar_init(&sm.s_full[i], 1); mbar_init(&sm.s_empty[i], 2 * kDGroup); }
    for (int i = 0; i < kYSlots; ++i) { mbar_init(&sm.y_full[i], 1); mbar_init(&sm.y_empty[i], kDGroups * kDGroup); }
    for (int i = 0; i < kSt; ++i) { mbar_init(&sm.full[i], kDGroup + 1); mbar_init(&sm.empty[i], 1); }
    mbar_init(&sm.acc_full, 1);
    mbar_init(&sm.folded, kEWarps);
    mbar_init(&sm.dotted, kEWarps);
    mbar_init(&sm.mma_done, 1);
    for (int i = 0; i < kQueue; ++i) { mbar_init(&sm.q_full[i], 1); mbar_init(&sm.q_empty[i], kQueueReaders); }
    fence_mbar_init();
    sm.fail = 0;
  }
  if (warp == kWarpMma) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.taddr)),
                 "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  uint32_t const tmem = sm.taddr;
  // FP16: the A scale of pair pi and flavour f from the tile copies' maxima,
  // x[1 - f] (rows S) and y[f] (rows Y): |D| <= 12 |Y| |S| <= 24 max|Y| max|S|
  auto a_scale = [&](uint32_t pi, int f) -> float {
    const float* tx = tb.x32[pi] + f32_tile_floats(geo.V);
    const float* ty = tb.y32 + f32_tile_floats(geo.V);
    return f16_scale(24.f * tx[1 - f] * ty[f]);
  };
  // the i-th unit of this CTA (>= nunits: no more), for a whole warp
  auto next = [&](int i, uint32_t& unit) -> bool {
    int const qs = i % kQueue;
    if (!wait_or_fail(&sm.q_full[qs], (uint32_t)((i / kQueue) & 1), fail)) return false;
    unit = *reinterpret_cast<volatile uint32_t*>(&sm.unit[qs]);
    __syncwarp();
    if (lane == 0) mbar_arrive(&sm.q_empty[qs]);
    return unit < nunits;
  };

  // issue tracking for the teardown after a failure
  int rows_issued_s = -1, rows_issued_y = -1;  // last S block / Y p-block use issued
  int b_issued = -1;
  int d_next = -1;  // D warps: the next chunk of this warp's group
  bool mma_any = false;

  if (warp == kWarpRows) {
    // ---- input rows ---------------------------------------------------------
    // per phase, in the order the D warps use them: the Y rows of p-block bp,
    // then the S rows of its three blocks. A wait here is for the ring slot
    // of a use two (Y) or three (S) steps back, whose readers need only rows
    // issued before it.
    if (lane == 0) {
      bool ok = true;
      uint32_t unit = blockIdx.x;
#pragma unroll 1
      for (int i = 0; ok; ++i) {
        int const qs = i % kQueue;
        if (!wait_or_fail(&sm.q_empty[qs], (uint32_t)(((i / kQueue) & 1) ^ 1), fail)) break;
        *reinterpret_cast<volatile uint32_t*>(&sm.unit[qs]) = unit;
        mbar_arrive(&sm.q_full[qs]);
        if (unit >= nunits) break;
        uint32_t const pi = unit / ntiles, tile = unit - pi * ntiles;
        // the next unit: drawn while this one's rows are issued
        unit = gridDim.x + atomicAdd(next_unit, 1u);
        const float* __restrict__ x32 = tb.x32[pi];
#pragma unroll 1
        for (int P = 2 * i; ok && P < 2 * i + 2; ++P) {
          int const f = P & 1;
#pragma unroll 1
          for (int bp = 0; ok && bp < 3; ++bp) {
#pragma unroll 1
            for (int h = 0; ok && h < 2; ++h) {
              int const uy = (P * 3 + bp) * 2 + h, ys = uy % kYSlots;
              if (!wait_or_fail(&sm.y_empty[ys], (uint32_t)(((uy / kYSlots) & 1) ^ 1), fail)) { ok = false; break; }
              fence_proxy_async_smem();
              mbar_arrive_expect_tx(&sm.y_full[ys], kYRows * kRowBytes);
              for (int r = 0; r < kYRows; ++r)
                bulk_g2s(sm.Y[ys][r], row_ptr(y32, f, 4 * bp + 2 * h + r, tile), kRowBytes, &sm.y_full[ys]);
              rows_issued_y = uy;
            }
#pragma unroll 1
            for (int bq = 0; ok && bq < kBlocksQ; ++bq) {
              int const us = P * kBlocks + bp * kBlocksQ + bq, ss = us % kSGroups;
              if (!wait_or_fail(&sm.s_empty[ss], (uint32_t)(((us / kSGroups) & 1) ^ 1), fail)) { ok = false; break; }
              fence_proxy_async_smem();
              mbar_arrive_expect_tx(&sm.s_full[ss], kRowsPerGroup * kRowBytes);
              for (int r = 0; r < kRowsPerGroup; ++r)
                bulk_g2s(sm.S[ss][r], row_ptr(x32, 1 - f, 4 * bq + r, tile), kRowBytes, &sm.s_full[ss]);
              rows_issued_s = us;
            }
          }
        }
      }
    }
  } else if (warp == kWarpB) {
    // ---- B chunks -------------------------------------------------------------
    constexpr int kBP = OpT<kF16>::kBParts;
    int bc = 0;
    bool ok = true;
    uint32_t unit;
#pragma unroll 1
    for (int i = 0; ok && next(i, unit); ++i) {
      uint32_t const pi = unit / ntiles;
#pragma unroll 1
      for (int f = 0; ok && f < 2; ++f) {
        const unsigned char* src =
            static_cast<const unsigned char*>(btu) + ((size_t)pi * 2 + f) * kChunks * kBP * Sm::kBPartB;
#pragma unroll 1
        for (int c = 0; c < kChunks; ++c, ++bc) {
          int const st = bc % kSt;
          if (!wait_or_fail(&sm.empty[st], (uint32_t)(((bc / kSt) & 1) ^ 1), fail)) { ok = false; break; }
          if (lane == 0) {
            fence_proxy_async_smem();
            mbar_arrive_expect_tx(&sm.full[st], kBP * Sm::kBPartB);
            bulk_g2s(sm.B[st][0], src + (size_t)c * kBP * Sm::kBPartB, kBP * Sm::kBPartB, &sm.full[st]);
          }
          __syncwarp();
          b_issued = bc;
        }
      }
    }
  } else if (warp == kWarpMma) {
    // ---- MMA issue ----------------------------------------------------------------
    // The tensor pipe runs the four FP16 MMAs of a chunk in about 330 cycles,
    // so the issuing warp's own per-chunk work has to stay well below that: the
    // whole warp walks the loop and waits, so that its control flow and the
    // descriptors are uniform, and one elected lane issues; the stage
    // descriptors differ only in their start address (bits 0-13, in 16-byte
    // units, no carry below 256 KB), so they are formed once and advanced by
    // constants; ring positions and phases are counters.
    {
      uint64_t const a_desc0 = sdesc(smem_u32(sm.A[0][0]), (kM / 8) * 128, 128);
      uint64_t const b_desc0 = sdesc(smem_u32(sm.B[0][0]), (kBtN / 8) * 128, 128);
      // in 16-byte units: stage to stage, hi to lo part, and (TF32, two
      // k-steps of 8 per chunk) k-step to k-step: two core columns, 2*16*128
      // and 2*20*128 bytes. FP16: one k-step of 16 per chunk (the chunk's two
      // core columns of 8 k)
      constexpr uint64_t kAStage16 = 2 * Sm::kAPartB / 16, kALo16 = Sm::kAPartB / 16, kAK16 = 2 * (kM / 8) * 128 / 16;
      constexpr uint64_t kBStage16 = OpT<kF16>::kBParts * Sm::kBPartB / 16, kBLo16 = Sm::kBPartB / 16,
                         kBK16 = 2 * (kBtN / 8) * 128 / 16;
      int as = 0;
      uint32_t aph = 0;
      uint32_t const dc = tmem + kCorrCol;
      bool ok = true;
      uint32_t unit = 0;
#pragma unroll 1
      for (int P = 0; ok; ++P) {
        if ((P & 1) == 0 && !next(P >> 1, unit)) break;
        // first half into main buffer P&1 (phase P-1's second half, free once
        // folded), second half into buffer (P+1)&1 (free once dotted)
        if (!wait_or_fail(&sm.folded, (uint32_t)((P & 1) ^ 1), fail)) break;
        tc_fence_after();
        uint32_t const d0 = tmem + (uint32_t)((P & 1) * kBtN), d1 = tmem + (uint32_t)(((P + 1) & 1) * kBtN);
#pragma unroll 1
        for (int c = 0; c < kChunks; ++c) {
          if (c == kHalf) {
            if (!wait_or_fail(&sm.dotted, (uint32_t)((P & 1) ^ 1), fail)) { ok = false; break; }
            tc_fence_after();
          }
          if (!wait_or_fail(&sm.full[as], aph, fail)) {
            ok = false;
            break;
          }
          tc_fence_after();
          uint32_t const d = c < kHalf ? d0 : d1;
          uint64_t const ahi = a_desc0 + (uint64_t)as * kAStage16, bhi = b_desc0 + (uint64_t)as * kBStage16;
          // hi.hi into the main buffer, hi.lo and lo.hi into the correction
          // accumulator
          if constexpr (kF16) {
            mma_chunk_f16(d, dc, ahi, ahi + kALo16, bhi, kBLo16, (c != 0 && c != kHalf) ? 1u : 0u, c ? 1u : 0u,
                          &sm.empty[as]);
          } else {
            if (elect_one()) {
              mma_tf32(d, ahi, bhi, (c != 0 && c != kHalf) ? 1u : 0u);
              mma_tf32(dc, ahi, bhi + kBLo16, c ? 1u : 0u);
              mma_tf32(dc, ahi + kALo16, bhi, 1u);
              mma_tf32(d, ahi + kAK16, bhi + kBK16, 1u);
              mma_tf32(dc, ahi + kAK16, bhi + kBK16 + kBLo16, 1u);
              mma_tf32(dc, ahi + kAK16 + kALo16, bhi + kBK16, 1u);
              mma_commit(&sm.empty[as]);  // frees the A and the B stage
            }
            __syncwarp();
          }
          mma_any = true;
          if (++as == kSt) { as = 0; aph ^= 1u; }
        }
        if (!ok) break;
        if (elect_one()) mma_commit(&sm.acc_full);
        __syncwarp();
      }
    }
  } else if (warp < kWarpE0) {
    // ---- D formation ----------------------------------------------------------------
    int const dw = warp == 2 ? 0 : warp - 3;    // 0 .. 11
    int const grp = dw / kDGroup;  // chunks c = grp, grp + 3, ...
    int const j = dw % kDGroup;    // the chunk's j-th pair of (p, q)
    d_next = grp;
    int const s = lane;
    bool ok = true;
    uint32_t unit = 0, last_pi = 0xFFFFFFFFu;
    int nvalid = 0;
    float ascale0 = 1.f, ascale1 = 1.f;
#pragma unroll 1
    for (int P = 0; ok; ++P) {
      if ((P & 1) == 0) {
        if (!next(P >> 1, unit)) break;
        uint32_t const pi = unit / ntiles, tile = unit - pi * ntiles;
        nvalid = (int)min((long long)kSites, geo.V - (long long)tile * kSites);
        if (kF16 && pi != last_pi) {
          ascale0 = a_scale(pi, 0);
          ascale1 = a_scale(pi, 1);
          last_pi = pi;
        }
      }
#pragma unroll 1
      for (int c = grp; c < kChunks; c += kDGroups) {
        // chunk c is half c & 1 of block b = (bp, bq): this warp's
        // pair is p = 4 bp + 2 (c & 1) + j/2 (row p_in of the Y half) and
        // q = 4 bq + q_in, q_in + 1 (rows of the S group), q_in = 2 (j & 1)
        int const b = c >> 1, bp = b / kBlocksQ, bq = b - bp * kBlocksQ;
        int const uy = (P * 3 + bp) * 2 + (c & 1), ys = uy % kYSlots;
        int const us = P * kBlocks + b, ss = us % kSGroups;
        ok = ok && wait_or_fail(&sm.y_full[ys], (uint32_t)((uy / kYSlots) & 1), fail);
        ok = ok && wait_or_fail(&sm.s_full[ss], (uint32_t)((us / kSGroups) & 1), fail);
        int const ac = P * kChunks + c, as = ac % kSt;
        if (!ok || !wait_or_fail(&sm.empty[as], (uint32_t)(((ac / kSt) & 1) ^ 1), fail)) { ok = false; break; }
        int const p_in = j >> 1, q_in = 2 * (j & 1);  // rows of the Y half and of the S group
        // k = 4j .. 4j+3 of the chunk, row (mu*32 + s). TF32: core column j,
        // the whole 16-byte row; FP16: core column j/2, its half j&1 (8 bytes)
        unsigned char* Ahi = sm.A[as][0] + (kF16 ? (j >> 1) * 2048 + s * 16 + 8 * (j & 1) : j * 2048 + s * 16);
        unsigned char* Alo = sm.A[as][1] + (kF16 ? (j >> 1) * 2048 + s * 16 + 8 * (j & 1) : j * 2048 + s * 16);
        if (s < nvalid) {
          float y[24];
          {
            const float* Yr = sm.Y[ys][p_in] + f32_tile_off(s, 0);
            float const sc = kF16 ? ((P & 1) ? ascale1 : ascale0) : 1.f;  // FP16: D scaled through Y
#pragma unroll
            for (int c4 = 0; c4 < 6; ++c4) {
              float4 const a = *reinterpret_cast<const float4*>(Yr + c4 * 64);
              y[4 * c4] = sc * a.x; y[4 * c4 + 1] = sc * a.y; y[4 * c4 + 2] = sc * a.z; y[4 * c4 + 3] = sc * a.w;
            }
          }
          float d[4][4];  // [mu][pq0 re, pq0 im, pq1 re, pq1 im]
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float* Sr = sm.S[ss][q_in + h] + f32_tile_off(s, 0);
            float x[24];
#pragma unroll
            for (int c4 = 0; c4 < 6; ++c4) {
              float4 const bb = *reinterpret_cast<const float4*>(Sr + c4 * 64);
              x[4 * c4] = bb.x; x[4 * c4 + 1] = bb.y; x[4 * c4 + 2] = bb.z; x[4 * c4 + 3] = bb.w;
            }
            // O[s1][s2] = sum_c Y[s1][c] conj(S[s2][c]) for s2 = s1^2 (a) and 3-s1 (b),
            // as packed FP32 pairs: with w = (Re Y, Im Y), U = sum_c w Re S and
            // V = sum_c w Im S (the S part broadcast), Re O = U.x + V.y and
            // Im O = U.y - V.x -- two packed FMAs per (c, s2). D_mu = sum_s1
            // i^((2 - g5g_ph(mu, s1)) & 3) O[s1][s2] (s2 = a for mu = 0, 3; b for
            // mu = 1, 2), i.e. D_0 = a0 + a1 - a2 - a3, D_3 = i (a1 + a3 - a0 - a2),
            // D_1 = -i (b0 + b1 + b2 + b3), D_2 = b0 - b1 + b2 - b3: the b
            // products are summed per parity of s1 inside the FMA chains.
            float a[4][2];
            float2 ube = make_float2(0.f, 0.f), vbe = ube, ubo = ube, vbo = ube;
#pragma unroll
            for (int s1 = 0; s1 < 4; ++s1) {
              float2 ua = make_float2(0.f, 0.f), va = ua;
#pragma unroll
              for (int cc = 0; cc < 3; ++cc) {
                float2 const w = make_float2(y[2 * (3 * s1 + cc)], y[2 * (3 * s1 + cc) + 1]);
                int const sa = 2 * (3 * (s1 ^ 2) + cc), sb = 2 * (3 * (3 - s1) + cc);
                ua = __ffma2_rn(w, make_float2(x[sa], x[sa]), ua);
                va = __ffma2_rn(w, make_float2(x[sa + 1], x[sa + 1]), va);
                if (s1 & 1) {
                  ubo = __ffma2_rn(w, make_float2(x[sb], x[sb]), ubo);
                  vbo = __ffma2_rn(w, make_float2(x[sb + 1], x[sb + 1]), vbo);
                } else {
                  ube = __ffma2_rn(w, make_float2(x[sb], x[sb]), ube);
                  vbe = __ffma2_rn(w, make_float2(x[sb + 1], x[sb + 1]), vbe);
                }
              }
              a[s1][0] = ua.x + va.y; a[s1][1] = ua.y - va.x;
            }
            float const ber = ube.x + vbe.y, bei = ube.y - vbe.x;
            float const bor = ubo.x + vbo.y, boi = ubo.y - vbo.x;
            float const a01r = a[0][0] + a[1][0], a01i = a[0][1] + a[1][1];
            float const a23r = a[2][0] + a[3][0], a23i = a[2][1] + a[3][1];
            float const a13r = a[1][0] + a[3][0], a13i = a[1][1] + a[3][1];
            float const a02r = a[0][0] + a[2][0], a02i = a[0][1] + a[2][1];
            d[0][2 * h] = a01r - a23r; d[0][2 * h + 1] = a01i - a23i;
            d[3][2 * h] = a02i - a13i; d[3][2 * h + 1] = a13r - a02r;  // i (a13 - a02)
            d[1][2 * h] = bei + boi;   d[1][2 * h + 1] = -(ber + bor);  // -i (be + bo)
            d[2][2 * h] = ber - bor;   d[2][2 * h + 1] = bei - boi;
          }
#pragma unroll
          for (int mu = 0; mu < 4; ++mu) {
            if constexpr (kF16) {
              uint2 hi, lo;
              f16_split2(d[mu][0], d[mu][1], hi.x, lo.x);
              f16_split2(d[mu][2], d[mu][3], hi.y, lo.y);
              *reinterpret_cast<uint2*>(Ahi + mu * 32 * 16) = hi;
              *reinterpret_cast<uint2*>(Alo + mu * 32 * 16) = lo;
            } else {
              float4 hi, lo;
              hi.x = tf32_round(d[mu][0]); hi.y = tf32_round(d[mu][1]);
              hi.z = tf32_round(d[mu][2]); hi.w = tf32_round(d[mu][3]);
              lo.x = tf32_round(d[mu][0] - hi.x); lo.y = tf32_round(d[mu][1] - hi.y);
              lo.z = tf32_round(d[mu][2] - hi.z); lo.w = tf32_round(d[mu][3] - hi.w);
              *reinterpret_cast<float4*>(Ahi + mu * 32 * 16) = hi;
              *reinterpret_cast<float4*>(Alo + mu * 32 * 16) = lo;
            }
          }
        } else {
#pragma unroll
          for (int mu = 0; mu < 4; ++mu) {
            if constexpr (kF16) {
              *reinterpret_cast<uint2*>(Ahi + mu * 32 * 16) = make_uint2(0u, 0u);
              *reinterpret_cast<uint2*>(Alo + mu * 32 * 16) = make_uint2(0u, 0u);
            } else {
              *reinterpret_cast<float4*>(Ahi + mu * 32 * 16) = make_float4(0.f, 0.f, 0.f, 0.f);
              *reinterpret_cast<float4*>(Alo + mu * 32 * 16) = make_float4(0.f, 0.f, 0.f, 0.f);
            }
          }
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&sm.full[as]);
          d_next = ac + kDGroups;
          // two groups read each S block, in one chunk each; every group
          // reads each Y half, in one of its three chunks (bq = 0..2)
          mbar_arrive(&sm.s_empty[ss]);
          mbar_arrive(&sm.y_empty[ys]);
        }
      }
    }
  } else {
    // ---- epilogue -----------------------------------------------------------------------
    int const quad = warp & 3;  // the TMEM lanes this warp may access; mu = quad
    int const s = lane;
    uint32_t const lane_addr = tmem + ((uint32_t)(quad * 32) << 16);
    double const xu = args.xunit;
    SiteQ q;
    uint32_t unit = 0, pi = 0, tile = 0, last_pi = 0xFFFFFFFFu;
    float inv0 = 1.f, inv1 = 1.f;  // FP16: the inverse scales per flavour (powers of two)
    bool valid = false;
#pragma unroll 1
    for (int P = 0;; ++P) {
      if ((P & 1) == 0) {
        if (!next(P >> 1, unit)) break;
        pi = unit / ntiles;
        tile = unit - pi * ntiles;
        valid = (long long)tile * kSites + s < geo.V;
        if (pi != last_pi) {
          if constexpr (kF16) {
            inv0 = 1.f / (a_scale(pi, 0) * bscale[2 * pi]);
            inv1 = 1.f / (a_scale(pi, 1) * bscale[2 * pi + 1]);
          }
#pragma unroll
          for (int r = 0; r < 4; ++r)
            q.ym[r] = (float)(coord_map(mod_pos(tb.yv[pi][r], geo.global[r]), geo.global[r]) * xu);
          last_pi = pi;
        }
      }
      if (!kGeneric && (P & 1) == 0) {
        // the row's site data, for both flavours of the tile
        const int gsx[4] = {tb.gsx[pi][0], tb.gsx[pi][1], tb.gsx[pi][2], tb.gsx[pi][3]};
        const int yv[4] = {tb.yv[pi][0], tb.yv[pi][1], tb.yv[pi][2], tb.yv[pi][3]};
        const double* __restrict__ wq = args.w + (size_t)pi * geo.V * 3 * HLBL_QED_NW;
        long long const vv = valid ? (long long)tile * kSites + s : geo.V - 1;
        int rel[4];
        rel_coords_fast(geo, gsx, vv, rel);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          q.xm[r] = (float)(coord_map(rel[r], geo.global[r]) * xu);
          q.xmy[r] = (float)(coord_map_diff(rel[r], yv[r], geo.global[r]) * xu);
          q.zh[r] = (float)coord_map_zerohalf(rel[r], geo.global[r]);
        }
#pragma unroll
        for (int e = 0; e < 3; ++e)
#pragma unroll
          for (int k = 0; k < HLBL_QED_NW; ++k) q.w[e][k] = (float)wq[((size_t)vv * 3 + e) * HLBL_QED_NW + k];
      }
      if (kGeneric && (P & 1) == 0) {
        // the tile's coefficients of this row quadrant (20 KB) towards L2 while the
        // accumulators fill: read from HBM they made the dot, which the next phase
        // waits for, 4 % of the kernel longer
        const float* c = static_cast<const float*>(args.coef) + (size_t)pi * args.coef_stride +
                         coef32_index((long long)tile * kSites, quad, 0);
#pragma unroll
        for (int l = 0; l < kSites * kBtN / 32; l += 32)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(c + (l + lane) * 32));
      }
      if (!wait_or_fail(&sm.acc_full, (uint32_t)(P & 1), fail)) break;
      tc_fence_after();
      uint32_t const c0 = (uint32_t)((P & 1) * kBtN), c1 = (uint32_t)(((P + 1) & 1) * kBtN);
      // fold the second half and the corrections into the first half
#pragma unroll 1
      for (int jj = 0; jj < 10; ++jj) {
        float m[16], h[16], k[16];
        tmem_ld16(lane_addr + c0 + 16 * jj, m);
        tmem_ld16(lane_addr + c1 + 16 * jj, h);
        tmem_ld16(lane_addr + kCorrCol + 16 * jj, k);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i) m[i] = (m[i] + h[i]) + k[i];
        tmem_st16(lane_addr + c0 + 16 * jj, m);
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.folded);
      tc_fence_after();
      float a;
      if constexpr (kGeneric) {
        // the row (mu = quad, site s of the tile); pad sites' coefficients are zero
        const float* __restrict__ cg = static_cast<const float*>(args.coef) + (size_t)pi * args.coef_stride;
        a = epilogue_row_generic(lane_addr, c0, cg + coef32_index((long long)tile * kSites, quad, 0) + (size_t)s * 4);
      } else {
        switch (quad) {
          case 0: a = epilogue_row<0>(lane_addr, c0, q); break;
          case 1: a = epilogue_row<1>(lane_addr, c0, q); break;
          case 2: a = epilogue_row<2>(lane_addr, c0, q); break;
          default: a = epilogue_row<3>(lane_addr, c0, q); break;
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.dotted);
      if constexpr (kF16) a *= (P & 1) ? inv1 : inv0;  // a power of two: exact
      // the quadrant's sum for this (tile, flavour), in a fixed order
      double v = valid ? -(double)a : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      if (lane == 0) tsum[((size_t)unit * 2 + (P & 1)) * kEWarps + quad] = v;
    }
  }

  // ---- teardown ----------------------------------------------------------------------------
  tc_fence_before();
  __syncthreads();
  if (*fail) {
    // let nothing this CTA started outlive it (each wait bounded)
    if (warp == kWarpRows && lane == 0) {
      for (int u = rows_issued_s - kSGroups + 1; u <= rows_issued_s; ++u)
        if (u >= 0) mbar_wait(&sm.s_full[u % kSGroups], (uint32_t)((u / kSGroups) & 1));
      for (int u = rows_issued_y - kYSlots + 1; u <= rows_issued_y; ++u)
        if (u >= 0) mbar_wait(&sm.y_full[u % kYSlots], (uint32_t)((u / kYSlots) & 1));
    }
    // the B copies complete the operand stages' barriers together with the D
    // warps, which may have stopped short: they make up their arrivals first
    // (a stage's barrier is in the phase of the last chunk issued into it)
    if (warp == kWarpB && lane == 0) sm.b_last = b_issued;
    __syncthreads();
    if (d_next >= 0 && lane == 0)
      for (int u = max(0, sm.b_last - kSt + 1); u <= sm.b_last; ++u)
        if (u >= d_next && (u - d_next) % kDGroups == 0) mbar_arrive(&sm.full[u % kSt]);
    if (warp == kWarpB && lane == 0)
      for (int u = max(0, b_issued - kSt + 1); u <= b_issued; ++u)
        mbar_wait(&sm.full[u % kSt], (uint32_t)((u / kSt) & 1));
    if (warp == kWarpMma && lane == 0 && mma_any) {
      mma_commit(&sm.mma_done);
      mbar_wait(&sm.mma_done, 0);
    }
    if (t == 0 && err) atomicExch(err, kErrWaitTimeout);
  }
  __syncthreads();
  tc_fence_after();
  if (warp == kWarpMma)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
}

// B operand of the tensor-core pass 2, from pass 1's sums dz with the gammas of
// both sides written out (bt_build_kernel's values of g_build_kernel's g). Per
// (pair, flavour) and chunk of 16 k, the 160 x 16 block of Bt^T in the K-major
// core-matrix layout. TF32 operands: hi and lo parts (core (kg, n/8) at
// (kg*20 + n/8)*128 bytes, row n%8 at 16 bytes, k%4 at 4 bytes). FP16 operands:
// the values times bscale as hi, lo and lo2 parts, each the rounding of the
// rest of the FP64 value (core (k/8, n/8) at (k/8*20 + n/8)*128 bytes, row n%8
// at 16 bytes, k%8 at 2 bytes); bscale per (pair, flavour) is 2^(15 - e) with
// 2^e above max |dz| (every Bt entry is a component of dz times a power of i),
// which every CTA finds for itself from the 2880 sums: one launch, where g, its
// maximum and the operand took three (8,192 sites,
// four pairs: 27 -> 16 us).
template <bool kF16>
__global__ void __launch_bounds__(256) btu_build_kernel(const double* __restrict__ dz, float* __restrict__ bscale,
                                                        void* __restrict__ btu) {
  int const fl = blockIdx.y, pi = blockIdx.z;
  int const i = blockIdx.x * 256 + threadIdx.x;
  dz += ((size_t)pi * 2 + fl) * kDzLen;
  double scale = 1.0;
  if constexpr (kF16) {
    // the largest magnitude by the high words' bits: the exponent is all that
    // the scale needs, and the integer pipe is 64 times the FP64 pipe
    __shared__ unsigned red[8];
    unsigned m = 0;
    for (int q = threadIdx.x; q < kDzLen; q += 256) m = max(m, (unsigned)__double2hiint(dz[q]) & 0x7FFFFFFFu);
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 8; ++w) m = max(m, red[w]);
    int const e2 = (int)(m >> 20) - 1022;  // the largest is below 2^e2 (zero, infinite, NaN, beyond FP32: no scale)
    float const sc = m == 0 || e2 > 127 ? 1.f : f16_scale_exp(e2);
    if (blockIdx.x == 0 && threadIdx.x == 0) bscale[pi * 2 + fl] = sc;
    scale = (double)sc;  // a power of two: exact
  }
  if (i >= kBtK * kBtN) return;
  int const k = i / kBtN, n = i % kBtN;
  // k within chunk c: 4 jj + 2 hh + e for the pair (p, q) the D formation
  // puts there (block b = c/2 of 4 p x 4 q, half c & 1)
  int const c = k / kKc, kl = k % kKc, jj = kl >> 2, hh = (kl >> 1) & 1, e = kl & 1;
  int const bb = c >> 1, bbp = bb / kBlocksQ, bbq = bb - bbp * kBlocksQ;
  int const p = 4 * bbp + 2 * (c & 1) + (jj >> 1), q = 4 * bbq + 2 * (jj & 1) + hh;
  int const lam = n & 3, nu = (n >> 2) & 3, j = n >> 4;
  // M[q][p] = i^(phases) dz[j][(s, c_q)][(gg5_src(nu, s_p), c_p)], s the spin
  // that gamma_lam gamma_5 takes s_q from (an involution)
  int const s2 = gg5_src(lam, q / 3), sp = p / 3;
  int const ph = (gg5_ph(lam, s2) + gg5_ph(nu, sp)) & 3;
  const double* v = dz + ((j * 12 + 3 * s2 + q % 3) * 12 + 3 * gg5_src(nu, sp) + p % 3) * 2;
  double re, im;
  mul_iph(ph, v[0], v[1], re, im);
  double const x = (e == 0 ? re : -im) * scale;
  if constexpr (kF16) {
    // x = f + g to 48 bits in FP32 (f64_to_f32: on the integer pipe), then the
    // parts from f and g in FP32 (f - hi and r - lo are exact)
    float const f = f64_to_f32(x), g = f64_to_f32(x - (double)f);
    __half const hi = __float2half_rn(f);
    float const r = f - __half2float(hi);
    __half const lo = __float2half_rn(r + g);
    __half const lo2 = __float2half_rn((r - __half2float(lo)) + g);
    int const off = ((kl >> 3) * (kBtN / 8) + (n >> 3)) * 64 + (n & 7) * 8 + (kl & 7);
    __half* out = static_cast<__half*>(btu) + (((size_t)pi * 2 + fl) * kChunks + c) * 3 * kBPart + off;
    out[0] = hi;
    out[kBPart] = lo;
    out[2 * kBPart] = lo2;
  } else {
    float const hi = __uint_as_float(tf32_rna((float)x));
    float const lo = __uint_as_float(tf32_rna((float)(x - (double)hi)));
    int const off = ((kl >> 2) * (kBtN / 8) + (n >> 3)) * 32 + (n & 7) * 4 + (kl & 3);
    float* out = static_cast<float*>(btu) + (((size_t)pi * 2 + fl) * kChunks + c) * 2 * kBPart + off;
    out[0] = hi;
    out[kBPart] = lo;
  }
}

// The pair's two sums from the tiles' (tsum[pair][tile][flavour][4]), in a fixed
// order: a thread takes every (32 gridDim.x)-th tile's value of one (flavour,
// quadrant), compensated, then the threads of a CTA, then the CTAs in order (by
// the last one to finish). It also readies the counters of the next call.
constexpr int kRedThreads = 256, kRedCtas = 64;
__global__ void __launch_bounds__(kRedThreads)
tile_reduce_kernel(const double* __restrict__ tsum, long long ntiles, double* __restrict__ part,
                   unsigned* __restrict__ next_unit, unsigned* __restrict__ done, PairBatch batch, int add) {
  __shared__ double rs[kRedThreads / 32][2], rc[kRedThreads / 32][2];
  static_assert(kRedThreads == 256 && kRedCtas == 64, "one warp adds eight warps' and 64 CTAs' sums");
  int const t = threadIdx.x, warp = t >> 5, lane = t & 31, pi = blockIdx.y;
  tsum += (size_t)pi * ntiles * 8;
  Neu a;
  for (long long i = (long long)blockIdx.x * kRedThreads + t; i < ntiles * 8; i += (long long)gridDim.x * kRedThreads)
    a.add(tsum[i]);
  // lanes: bits 0, 1 the quadrant, bit 2 the flavour, bits 3, 4 the tile
#pragma unroll
  for (int o : {16, 8, 2, 1}) {
    double const os = __shfl_xor_sync(0xffffffffu, a.s, o), oc = __shfl_xor_sync(0xffffffffu, a.c, o);
    a.add(os);
    a.c += oc;
  }
  if ((lane & ~4) == 0) {
    rs[warp][lane >> 2] = a.s;
    rc[warp][lane >> 2] = a.c;
  }
  __syncthreads();
  if (warp != 0) return;
  // the warps' sums: lane 2 w + f
  a = Neu();
  if (lane < 2 * (kRedThreads / 32)) {
    a.s = rs[lane >> 1][lane & 1];
    a.c = rc[lane >> 1][lane & 1];
  }
#pragma unroll
  for (int o : {8, 4, 2}) {
    double const os = __shfl_xor_sync(0xffffffffu, a.s, o), oc = __shfl_xor_sync(0xffffffffu, a.c, o);
    a.add(os);
    a.c += oc;
  }
  if (gridDim.x > 1) {
    double* const parts = part + (size_t)pi * kRedCtas * 4;
    if (lane < 2) {
      parts[blockIdx.x * 4 + lane * 2] = a.s;
      parts[blockIdx.x * 4 + lane * 2 + 1] = a.c;
      __threadfence();
    }
    __syncwarp();
    int last = 0;
    if (lane == 0) last = atomicAdd(done + pi, 1u) == gridDim.x - 1;
    if (!__shfl_sync(0xffffffffu, last, 0)) return;
    __threadfence();
    // the CTAs' sums: lane 2 i + f takes CTAs i, i + 16, i + 32, i + 48
    a = Neu();
    for (unsigned g = lane >> 1; g < gridDim.x; g += 16) {
      a.add(__ldcg(parts + g * 4 + (lane & 1) * 2));
      a.c += __ldcg(parts + g * 4 + (lane & 1) * 2 + 1);
    }
#pragma unroll
    for (int o : {16, 8, 4, 2}) {
      double const os = __shfl_xor_sync(0xffffffffu, a.s, o), oc = __shfl_xor_sync(0xffffffffu, a.c, o);
      a.add(os);
      a.c += oc;
    }
  }
  if (lane < 2) {
    double* out = batch.p[pi].out;
    if (add) out[lane] += a.get();
    else out[lane] = a.get();
  }
  if (lane == 0) {
    done[pi] = 0u;
    if (pi == 0) *next_unit = 0u;
  }
}

}  // namespace tc

size_t tc_smem_bytes() { return sizeof(tc::Smem); }
int tc_threads() { return tc::kThreads; }
size_t tc_btu_floats_per_pair() { return (size_t)2 * tc::kChunks * 2 * tc::kBPart; }

template <bool G, bool F>
static int tc_init_one(int& nb) {
  size_t const smem = sizeof(tc::SmemT<F>);
  cudaError_t e = cudaFuncSetAttribute(tc::p2tc_kernel<G, F>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return cuda_fail(e, "p2tc smem attribute");
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, tc::p2tc_kernel<G, F>, tc::kThreads, smem);
  if (e != cudaSuccess) return cuda_fail(e, "p2tc occupancy");
  if (nb < 1) return fail(HLBL_ECUDA, "p2tc kernel cannot be resident (smem %zu)", smem);
  return HLBL_OK;
}

int tc_init(int nsm, int& grid) {
  int nb = 0;
  if (int rc = tc_init_one<false, false>(nb)) return rc;
  if (int rc = tc_init_one<true, false>(nb)) return rc;
  if (int rc = tc_init_one<false, true>(nb)) return rc;
  if (int rc = tc_init_one<true, true>(nb)) return rc;
  // one CTA per SM: each allocates all 512 TMEM columns
  grid = nsm;
  return HLBL_OK;
}

void tc_launch_btu(const double* d_dz, int npairs, void* d_btu, bool f16, float* d_bscale, cudaStream_t st) {
  dim3 const gb((kBtK * kBtN + 255) / 256, 2, npairs);
  if (f16) tc::btu_build_kernel<true><<<gb, 256, 0, st>>>(d_dz, d_bscale, d_btu);
  else tc::btu_build_kernel<false><<<gb, 256, 0, st>>>(d_dz, d_bscale, d_btu);
}

void tc_launch_p2(int nsm, int npairs, cudaStream_t st, const TcBatch& tb, const Geometry& geo, const P2Args& a,
                  const void* d_btu, bool f16, const float* d_bscale, double* tsum, unsigned* next_unit, int* err) {
  long long const units = tc_tiles(geo.V) * npairs;
  int const gr = (int)(units < nsm ? units : nsm);
  if (f16) {
    size_t const smem = sizeof(tc::SmemT<true>);
    if (a.coef) tc::p2tc_kernel<true, true><<<gr, tc::kThreads, smem, st>>>(tb, geo, a, d_btu, d_bscale, npairs, tsum, next_unit, err);
    else tc::p2tc_kernel<false, true><<<gr, tc::kThreads, smem, st>>>(tb, geo, a, d_btu, d_bscale, npairs, tsum, next_unit, err);
  } else {
    size_t const smem = sizeof(tc::SmemT<false>);
    if (a.coef) tc::p2tc_kernel<true, false><<<gr, tc::kThreads, smem, st>>>(tb, geo, a, d_btu, d_bscale, npairs, tsum, next_unit, err);
    else tc::p2tc_kernel<false, false><<<gr, tc::kThreads, smem, st>>>(tb, geo, a, d_btu, d_bscale, npairs, tsum, next_unit, err);
  }
}

size_t tc_tsum_len(long long V, int npairs) { return (size_t)tc_tiles(V) * npairs * 2 * tc::kEWarps; }

void tc_launch_reduce(int npairs, cudaStream_t st, const Geometry& geo, const double* tsum, double* part,
                      unsigned* next_unit, unsigned* done, const PairBatch& b, int add) {
  long long const tiles = tc_tiles(geo.V);
  // 64 tiles' sums per CTA (two per thread), up to 64 CTAs
  int const g = (int)std::min<long long>(tc::kRedCtas, (tiles + 63) / 64);
  tc::tile_reduce_kernel<<<dim3(g, npairs), tc::kRedThreads, 0, st>>>(tsum, tiles, part, next_unit, done, b, add);
}

long long tc_tiles(long long V) { return (V + tc::kSites - 1) / tc::kSites; }

}  // namespace hg
