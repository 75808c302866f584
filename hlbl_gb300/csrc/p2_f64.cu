// p2_f64.cu -- the FP64 pass 2 (ker_4pt_contraction, cuda_lattice.cu:277-484)
// in the block-diagonal form of quat_basis.cuh: for several pairs on lattices too
// small for the digit products of p2_dig.cu, and where their work buffer cannot be had.
//
// What bounds it: the FP64 pipe (two lanes per SM and cycle here), so the
// kernel is laid out for few FP64 instructions and nothing else. Per site and
// flavour: the D formation 14.9 k (96 multiply-adds per (p, q) and 16 adds),
// the contraction 46.1 k multiply-adds (184.3 k in the direct form of one
// 288 x 160 product per mu), the dot 2.6 k; per site the 640 coefficients
// 11.5 k and their sums per chirality block 4.5 k. Measured (both flavours, one
// pair): 7.00 -> 2.39 ms at 8,192 sites, 545.7 -> 185 ms at 663,552, the FP64 pipe
// 90 % active; one flavour at 41,472 sites 19.9 -> 6.5 ms.
#include <cuda_runtime.h>

#include <cstdint>

#include "contract_kernels.cuh"
#include "hlbl_gb300.h"
#include "hlbl_internal.h"
#include "p2_f64.h"
#include "qed_entry.cuh"
#include "quat_basis.cuh"

namespace hg {
namespace p2d {

constexpr int kTS = 4;                   // sites per tile
constexpr int kThreads = 320;            // two flavours x 160 columns, or one flavour x two halves of the tile
constexpr int kRowD = kTS * 24 + 2;      // staged row: 16 bytes of padding against bank conflicts
template <int NF>
struct __align__(128) Smem {
  double stage[2 * NF * 12][kRowD];
  double D[kTS][NF][4][4][quat::kBlk * quat::kKb];  // [site][flavour][mu][b][blk*18 + k]
  double coef[kTS][4][kBtN];
  double cq[quat::kBlk][kTS][4][kBtN];              // coefficients of [b*40 + j*4 + a] per block
  double vec[kTS][12];                              // xm, x - y, zerohalf x
  double tab[kTS * 3][kQedTab + 1];
};
static_assert(sizeof(Smem<2>) + 1024 <= 232448, "FP64 pass-2 shared memory above the 227 KB a CTA may have");

// dz in the form of quat_basis.cuh, halved: dzq[pair][fl][blk][k][j*4 + a],
// k = (c_p*3 + c_q)*2 + e, the real part (e = 0) or minus the imaginary part
// of z_a. From pass 1's sums (dz), or from sums with the gammas inserted
// (g_dzu, g_dzsu: their nu = 0 copy is undone); then `bad` is set if the four
// copies are not each other's images, as the caller may pass any numbers.
__global__ void dzq_build_kernel(const double* __restrict__ dz, const double* __restrict__ g_dzu,
                                 const double* __restrict__ g_dzsu, int nf, double* __restrict__ dzq,
                                 int* __restrict__ bad) {
  int const fl = blockIdx.y, pi = blockIdx.z;
  int const i = blockIdx.x * blockDim.x + threadIdx.x;
  if (dz != nullptr) dz += ((size_t)pi * nf + fl) * kDzLen;
  // (j, ia, ib) of dz
  auto at = [&](int j, int ia, int ib, double v[2]) {
    if (dz != nullptr) {
      v[0] = dz[((j * 12 + ia) * 12 + ib) * 2];
      v[1] = dz[((j * 12 + ia) * 12 + ib) * 2 + 1];
      return;
    }
    // g[j][nu][ia][(s, c)] = i^gg5_ph(nu, s) dz[j][ia][(gg5_src(nu, s), c)]; gg5_src is an involution
    int const sp = gg5_src(0, ib / 3), c = ib % 3;
    const double* g = (j < 6 ? g_dzu + (size_t)j * 1152 : g_dzsu + (size_t)(j - 6) * 1152) + (ia * 12 + 3 * sp + c) * 2;
    mul_iph((4 - gg5_ph(0, sp)) & 3, g[0], g[1], v[0], v[1]);
  };
  if (dz == nullptr && bad != nullptr && i < kGLen / 2) {
    int const ib = i % 12, ia = (i / 12) % 12, nu = (i / 144) % 4, j = i / 576;
    const double* g = (j < 6 ? g_dzu + (size_t)j * 1152 : g_dzsu + (size_t)(j - 6) * 1152) + ((nu * 12 + ia) * 12 + ib) * 2;
    double v[2], re, im;
    at(j, ia, 3 * gg5_src(nu, ib / 3) + ib % 3, v);
    mul_iph(gg5_ph(nu, ib / 3), v[0], v[1], re, im);
    if (!(re == g[0] && im == g[1])) *bad = 1;
  }
  if (i >= quat::kLen || fl >= nf) return;
  int const col = i % quat::kCol, k = (i / quat::kCol) % quat::kKb, blk = i / (quat::kCol * quat::kKb);
  int const j = col >> 2, a = col & 3, e = k & 1, cq = (k >> 1) % 3, cp = (k >> 1) / 3;
  int const r0 = 3 * 2 * (1 - (blk & 1)) + cq, c0 = 3 * 2 * (1 - (blk >> 1)) + cp;  // spins 2(1-chi_q), 2(1-chi_p)
  double z[4][2], c[4][2];
  at(j, r0, c0, z[0]);
  at(j, r0, c0 + 3, z[1]);
  at(j, r0 + 3, c0, z[2]);
  at(j, r0 + 3, c0 + 3, z[3]);
  quat::components(z[0], z[1], z[2], z[3], c);
  double const re = a == 0 ? c[0][0] : (a == 1 ? c[1][0] : (a == 2 ? c[2][0] : c[3][0]));
  double const im = a == 0 ? c[0][1] : (a == 1 ? c[1][1] : (a == 2 ? c[2][1] : c[3][1]));
  dzq[((size_t)pi * nf + fl) * quat::kLen + i] = 0.5 * (e == 0 ? re : -im);
}

// Per CTA partials of pass 2 (p2_kernel's sums). A tile is four sites: two
// flavours' rows, their D in shared memory, then thread (fl, b, j, a) holds
// the 16 sums (site, mu) of one column over a block's 18 k, the D values
// broadcast and the column's dz read through L1. One stage: the next tile is
// fetched while this one is contracted (2 % of the time of the products).
// skip: return at once if *skip (the sums are then p2_kernel's).
template <int NF>
__global__ void __launch_bounds__(kThreads, 1)
p2f64_kernel(const double* __restrict__ y, PairBatch batch, Geometry geo, P2Args args,
             const double* __restrict__ dzq_all, double* __restrict__ partials, int* __restrict__ err,
             const int* __restrict__ skip) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  Smem<NF>& sm = *reinterpret_cast<Smem<NF>*>(smem_raw);
  __shared__ __align__(8) uint64_t s_bar;
  __shared__ int s_fail;
  __shared__ double s_red[kThreads / 32][2];
  if (skip != nullptr && *skip != 0) return;
  constexpr int nthr = kThreads, kSitesT = kTS * NF / 2;  // sites of a thread
  int const t = threadIdx.x;
  int const pi = blockIdx.y;
  const double* __restrict__ src = batch.p[pi].src;
  int const gsx[4] = {batch.p[pi].gsx[0], batch.p[pi].gsx[1], batch.p[pi].gsx[2], batch.p[pi].gsx[3]};
  int const yv[4] = {batch.p[pi].yv[0], batch.p[pi].yv[1], batch.p[pi].yv[2], batch.p[pi].yv[3]};
  const double* __restrict__ wq = args.w ? args.w + (size_t)pi * geo.V * 3 * HLBL_QED_NW : nullptr;
  double const xu = args.xunit;
  // S = src at flavour 1-f, Y = y at flavour f, f = f0 + fl; rows [S | Y][fl][12]
  auto issue = [&](long long s0) {
    uint32_t const bytes = (uint32_t)min((long long)kTS, geo.V - s0) * 192u;
    mbar_arrive_expect_tx(&s_bar, bytes * 2 * NF * 12);
    for (int row = 0; row < 2 * NF * 12; ++row) {
      int const which = row / (NF * 12), fl = (row / 12) % NF, ia = row % 12;
      int const f = which == 0 ? 1 - args.f0 - fl : args.f0 + fl;
      bulk_g2s(sm.stage[row], (which == 0 ? src : y) + ((size_t)(f * 12 + ia) * geo.V + s0) * 24, bytes, &s_bar);
    }
  };
  if (t == 0) {
    mbar_init(&s_bar, 1);
    fence_mbar_init();
    s_fail = 0;
  }
  __syncthreads();

  int const fl = NF == 2 ? t / 160 : 0, st0 = NF == 2 ? 0 : (t / 160) * kSitesT;
  int const col = t % 160, b = col / quat::kCol, ja = col % quat::kCol;
  const double* __restrict__ B = dzq_all + ((size_t)pi * NF + fl) * quat::kLen + ja;
  Neu run;
  long long const ntiles = (geo.V + kTS - 1) / kTS;
  long long tile = blockIdx.x;
  if (t == 0 && tile < ntiles) issue(tile * kTS);
  uint32_t parity = 0;
  for (; tile < ntiles; tile += gridDim.x, parity ^= 1u) {
    long long const s0 = tile * kTS;
    int const nvalid = (int)min((long long)kTS, geo.V - s0);
    // per site: xm, x - y (minimum image) and the zerohalf weights
    if (t < kTS * 4) {
      int const s = t >> 2, r = t & 3;
      int rel[4];
      rel_coords_fast(geo, gsx, min(s0 + s, geo.V - 1), rel);
      sm.vec[s][r] = coord_map(rel[r], geo.global[r]) * xu;
      sm.vec[s][4 + r] = coord_map_diff(rel[r], yv[r], geo.global[r]) * xu;
      sm.vec[s][8 + r] = (double)coord_map_zerohalf(rel[r], geo.global[r]);
    }
    __syncthreads();
    if (args.coef) {
      // generic QED path: the coefficients of the tile's sites (zero past the end)
      const double* cg = static_cast<const double*>(args.coef) + (size_t)pi * args.coef_stride;
      for (int it = t; it < kTS * kCoefPerSite; it += nthr) {
        long long const site = s0 + it / kCoefPerSite;
        (&sm.coef[0][0][0])[it] = site < geo.V ? __ldg(cg + (size_t)s0 * kCoefPerSite + it) : 0.0;
      }
    } else {
      // the tensor's factors per (site, evaluation): e = 0: K(x, y), 1: K(y, x), 2: K(x, x - y)
      for (int it = t; it < kTS * 3 * kQedTab; it += nthr) {
        int const se = it / kQedTab, i = it % kQedTab, s = se / 3, e = se % 3;
        const double* xm = sm.vec[s];
        double ym[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) ym[r] = coord_map(mod_pos(yv[r], geo.global[r]), geo.global[r]) * xu;
        double const v = qed_tab_value(i, e == 1 ? ym : xm, e == 0 ? ym : (e == 1 ? xm : xm + 4),
                                       wq + (size_t)(min(s0 + s, geo.V - 1) * 3 + e) * HLBL_QED_NW);
        sm.tab[se][i] = v;
      }
      __syncthreads();
      // coefficients (site-dependent, flavour-independent)
      for (int it = t; it < kTS * kCoefPerSite; it += nthr) {
        int const s = it / kCoefPerSite, mu = (it / kBtN) & 3, n = it % kBtN;
        int const lam = n & 3, nu = (n >> 2) & 3, j = n >> 4;
        const double* q1 = sm.tab[s * 3];
        const double* q2 = sm.tab[s * 3 + 1];
        const double* q3 = sm.tab[s * 3 + 2];
        double cf;
        if (j < 6) {
          int const r = comb_rho(j), g = comb_sigma(j);
          cf = qed_entry_tab(q1, j, r, g, mu, nu, lam) + qed_entry_tab(q2, j, r, g, nu, mu, lam) - qed_entry_tab(q3, j, r, g, lam, nu, mu);
        } else {
          // sum_k E3[k][lam][nu][mu] (zh_rho_k [sigma_k = tau] - zh_sigma_k [rho_k = tau])
          int const tau = j - 6;
          cf = 0.0;
          for (int o = 0; o < 4; ++o) {
            if (o == tau) continue;
            int const r = min(o, tau), g = max(o, tau), k = r == 0 ? g - 1 : (r == 1 ? g + 1 : 5);
            cf = fma(flip_sign(sm.vec[s][8 + o], tau < o ? 1u : 0u), qed_entry_tab(q3, k, r, g, lam, nu, mu), cf);
          }
        }
        sm.coef[s][mu][n] = s < nvalid ? cf : 0.0;
      }
    }
    // the tile's blocks have landed
    if (!mbar_wait(&s_bar, parity)) s_fail = 1;
    __syncthreads();
    if (s_fail) break;
    // the coefficients' sums per chirality block: task (site, mu, j, class)
    for (int it = t; it < kTS * 4 * 10 * 4; it += nthr) {
      int const kap = it & 3, j = (it >> 2) % 10, smu = it / 40, mu = smu & 3, s = smu >> 2;
      double c[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) c[m] = sm.coef[s][mu][16 * j + 4 * m + (m ^ kap)];
#pragma unroll
      for (int bb = 0; bb < 4; ++bb) {
        double out[4];
        quat::class_sums(c, kap, bb ^ kap, bb, out);
#pragma unroll
        for (int blk = 0; blk < 4; ++blk) sm.cq[blk][s][mu][bb * quat::kCol + 4 * j + (bb ^ kap)] = out[blk];
      }
    }
    // D_mu's quaternion components: task (site, fl, chi_p, chi_q, c_p, c_q)
    for (int it = t; it < kTS * NF * 36; it += nthr) {
      int const s = it % kTS, f = (it / kTS) % NF, tk = it / (kTS * NF);
      int const blk = tk / 9, cp = (tk % 9) / 3, cq = tk % 3;
      double* Do = &sm.D[s][f][0][0][blk * quat::kKb + 2 * (tk % 9)];
      if (s >= nvalid) {
#pragma unroll
        for (int mb = 0; mb < 16; ++mb) *reinterpret_cast<double2*>(Do + mb * (quat::kBlk * quat::kKb)) = make_double2(0.0, 0.0);
        continue;
      }
      double X[4][4][2];  // [mu][2 i + k]
#pragma unroll
      for (int ik = 0; ik < 4; ++ik) {
        int const p = 3 * (2 * (blk >> 1) + (ik >> 1)) + cp, q = 3 * (2 * (blk & 1) + (ik & 1)) + cq;
        const double2* S = reinterpret_cast<const double2*>(&sm.stage[f * 12 + q][s * 24]);
        const double2* Y = reinterpret_cast<const double2*>(&sm.stage[(NF + f) * 12 + p][s * 24]);
        // O[s1][s2] = sum_c Y[s1][c] conj(S[s2][c]): al = O02 - O31, be = O13 - O20,
        // ev = O03 + O21, od = O12 + O30; D_0 = al + be, D_3 = i (be - al),
        // D_1 = -i (ev + od), D_2 = ev - od
        double ar = 0, ai = 0, br = 0, bi = 0, er = 0, ei = 0, orr = 0, oi = 0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          double2 const y0 = Y[c], y1 = Y[3 + c], y2 = Y[6 + c], y3 = Y[9 + c];
          double2 const x0 = S[c], x1 = S[3 + c], x2 = S[6 + c], x3 = S[9 + c];
          ar += y0.x * x2.x; ar += y0.y * x2.y; ar -= y3.x * x1.x; ar -= y3.y * x1.y;
          ai += y0.y * x2.x; ai -= y0.x * x2.y; ai -= y3.y * x1.x; ai += y3.x * x1.y;
          br += y1.x * x3.x; br += y1.y * x3.y; br -= y2.x * x0.x; br -= y2.y * x0.y;
          bi += y1.y * x3.x; bi -= y1.x * x3.y; bi -= y2.y * x0.x; bi += y2.x * x0.y;
          er += y0.x * x3.x; er += y0.y * x3.y; er += y2.x * x1.x; er += y2.y * x1.y;
          ei += y0.y * x3.x; ei -= y0.x * x3.y; ei += y2.y * x1.x; ei -= y2.x * x1.y;
          orr += y1.x * x2.x; orr += y1.y * x2.y; orr += y3.x * x0.x; orr += y3.y * x0.y;
          oi += y1.y * x2.x; oi -= y1.x * x2.y; oi += y3.y * x0.x; oi -= y3.x * x0.y;
        }
        X[0][ik][0] = ar + br;  X[0][ik][1] = ai + bi;
        X[3][ik][0] = ai - bi;  X[3][ik][1] = br - ar;
        X[1][ik][0] = ei + oi;  X[1][ik][1] = -(er + orr);
        X[2][ik][0] = er - orr; X[2][ik][1] = ei - oi;
      }
#pragma unroll
      for (int mu = 0; mu < 4; ++mu) {
        double c[4][2];
        quat::components(X[mu][0], X[mu][1], X[mu][2], X[mu][3], c);
#pragma unroll
        for (int bb = 0; bb < 4; ++bb)
          *reinterpret_cast<double2*>(Do + (mu * 4 + bb) * (quat::kBlk * quat::kKb)) = make_double2(c[bb][0], c[bb][1]);
      }
    }
    __syncthreads();
    if (t == 0 && tile + gridDim.x < ntiles) {
      fence_proxy_async_smem();
      issue((tile + gridDim.x) * kTS);
    }
    // the contraction and the dot
    double part = 0.0;
#pragma unroll 1
    for (int blk = 0; blk < quat::kBlk; ++blk) {
      double acc[kSitesT][4];
#pragma unroll
      for (int s = 0; s < kSitesT; ++s)
#pragma unroll
        for (int mu = 0; mu < 4; ++mu) acc[s][mu] = 0.0;
      const double* Bk = B + blk * quat::kKb * quat::kCol;
      const double* Dk = &sm.D[st0][fl][0][b][blk * quat::kKb];
#pragma unroll 3
      for (int k = 0; k < quat::kKb; k += 2) {
        double const b0 = __ldg(Bk + k * quat::kCol), b1 = __ldg(Bk + (k + 1) * quat::kCol);
#pragma unroll
        for (int s = 0; s < kSitesT; ++s)
#pragma unroll
          for (int mu = 0; mu < 4; ++mu) {
            double2 const d = *reinterpret_cast<const double2*>(Dk + (s * NF * 16 + mu * 4) * (quat::kBlk * quat::kKb) + k);
            acc[s][mu] = fma(d.x, b0, acc[s][mu]);
            acc[s][mu] = fma(d.y, b1, acc[s][mu]);
          }
      }
#pragma unroll
      for (int s = 0; s < kSitesT; ++s)
#pragma unroll
        for (int mu = 0; mu < 4; ++mu) part = fma(sm.cq[blk][st0 + s][mu][col], acc[s][mu], part);
    }
    run.add(-part);
    __syncthreads();  // everything but the stage is rewritten in the next iteration
  }
  if (s_fail) {
    // the copy that was waited for is the only one in flight: let it land
    // before the CTA exits (bounded, as everything else)
    if (t == 0) {
      if (err) atomicExch(err, kErrWaitTimeout);
      mbar_wait(&s_bar, parity);
    }
    return;
  }
  // block reduction per flavour in a fixed order, as p2_kernel's
  Neu v = run;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    double const os = __shfl_down_sync(0xffffffffu, v.s, o);
    double const oc = __shfl_down_sync(0xffffffffu, v.c, o);
    v.add(os);
    v.c += oc;
  }
  if ((t & 31) == 0) { s_red[t >> 5][0] = v.s; s_red[t >> 5][1] = v.c; }
  __syncthreads();
  if (t < NF) {
    Neu s;
    constexpr int kW = kThreads / 32 / NF;  // warps of a flavour
    for (int w = t * kW; w < (t + 1) * kW; ++w) { s.add(s_red[w][0]); s.c += s_red[w][1]; }
    partials[((size_t)pi * gridDim.x + blockIdx.x) * NF + t] = s.get();
  }
}

}  // namespace p2d

template <int NF>
static int p2f64_init_t(int nsm, int& grid) {
  size_t const smem = sizeof(p2d::Smem<NF>);
  cudaError_t e = cudaFuncSetAttribute(p2d::p2f64_kernel<NF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return cuda_fail(e, "p2f64 smem attribute");
  int nb = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, p2d::p2f64_kernel<NF>, p2d::kThreads, smem);
  if (e != cudaSuccess) return cuda_fail(e, "p2f64 occupancy");
  if (nb < 1) return fail(HLBL_ECUDA, "p2f64 kernel cannot be resident (smem %zu)", smem);
  grid = nb * nsm;
  return HLBL_OK;
}

int p2f64_init(int nsm, int grid[2]) {
  if (int rc = p2f64_init_t<1>(nsm, grid[0])) return rc;
  return p2f64_init_t<2>(nsm, grid[1]);
}

size_t p2f64_dzq_len() { return quat::kLen; }
long long p2f64_tiles(long long V) { return (V + p2d::kTS - 1) / p2d::kTS; }

void p2f64_launch_dzq(const double* dz, const double* g_dzu, const double* g_dzsu, int nf, int npairs, double* dzq,
                      int* bad, cudaStream_t st) {
  int const n = bad != nullptr ? kGLen / 2 : quat::kLen;
  p2d::dzq_build_kernel<<<dim3((n + 127) / 128, nf, npairs), 128, 0, st>>>(dz, g_dzu, g_dzsu, nf, dzq, bad);
}

void p2f64_launch(int nf, int grid, cudaStream_t st, const double* y, const PairBatch& b, const Geometry& geo,
                  const P2Args& a, const double* dzq, double* partials, int* err, const int* skip) {
  if (nf == 2)
    p2d::p2f64_kernel<2><<<dim3(grid, b.n), p2d::kThreads, sizeof(p2d::Smem<2>), st>>>(y, b, geo, a, dzq, partials, err, skip);
  else
    p2d::p2f64_kernel<1><<<dim3(grid, b.n), p2d::kThreads, sizeof(p2d::Smem<1>), st>>>(y, b, geo, a, dzq, partials, err, skip);
}

}  // namespace hg
