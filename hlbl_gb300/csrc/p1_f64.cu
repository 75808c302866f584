// p1_f64.cu -- the FP64 pass 1 (ker_dzu_dzsu, cuda_lattice.cu:160-262).
//
// Thread (fl, ia, ib) owns dzu[k][ia][ib] and dzsu[s][ia][ib] of flavour
// f = f0 + fl, as in p1_kernel. What bounds it is the FP64 pipe, so it is laid
// out for few FP64 instructions per site and thread: the eight spin-block
// products in four sums of two blocks each (96 multiply-adds, all that the four
// X_sigma need), and, as the zerohalf weights zh_0..zh_2 are constant along a
// run of sites in z, only the run's sums of the products and of zh_3 times them
// (8 adds and 8 multiply-adds; 56 with all ten weighted sums per site). The
// runs' sums go into the ten results at the end of each run, those into the
// compensated sums every kFlushTiles tiles. Measured (both flavours, one pair):
// 85.3 -> 42 ms at 663,552 sites, 1.11 -> 0.57 ms at 8,192.
#include <cuda_runtime.h>

#include <cstdint>

#include "contract_kernels.cuh"
#include "hlbl_gb300.h"
#include "hlbl_internal.h"
#include "p1_f64.h"

namespace hg {
namespace p1d {

constexpr int kTS = 8;                 // sites per tile
constexpr int kRow = kTS * 24 + 2;     // staged row: 16 bytes of padding against bank conflicts
constexpr int kFlushTiles = 4;         // tiles per addition into the compensated sums
template <int NF>
struct __align__(128) Smem {
  double stage[2][2 * NF * 12][kRow];
  double zh[2][kTS][4];
};

template <int NF>
__global__ void __launch_bounds__(NF * 144, NF == 1 ? 2 : 1)
p1f64_kernel(const double* __restrict__ y, PairBatch batch, Geometry geo, int f0, double* __restrict__ partials,
             int* __restrict__ err) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  Smem<NF>& sm = *reinterpret_cast<Smem<NF>*>(smem_raw);
  __shared__ __align__(8) uint64_t s_bar[2];
  __shared__ int s_fail;
  int const t = threadIdx.x, pi = blockIdx.y;
  const double* __restrict__ src = batch.p[pi].src;
  int const gsx[4] = {batch.p[pi].gsx[0], batch.p[pi].gsx[1], batch.p[pi].gsx[2], batch.p[pi].gsx[3]};
  int const fl = t / 144, ia = (t % 144) / 12, ib = t % 12;
  // rows [src | y][fl][12]: src flavour f0 + fl, y flavour 1 - (f0 + fl)
  auto issue = [&](long long tile, int st) {
    long long const s0 = tile * kTS;
    uint32_t const bytes = (uint32_t)min((long long)kTS, geo.V - s0) * 192u;
    mbar_arrive_expect_tx(&s_bar[st], bytes * 2 * NF * 12);
    for (int row = 0; row < 2 * NF * 12; ++row) {
      int const which = row / (NF * 12), f = (row / 12) % NF, i = row % 12;
      int const ff = which == 0 ? f0 + f : 1 - f0 - f;
      bulk_g2s(sm.stage[st][row], (which == 0 ? src : y) + ((size_t)(ff * 12 + i) * geo.V + s0) * 24, bytes, &s_bar[st]);
    }
  };
  auto zh_fill = [&](long long tile, int buf) {
    for (int s = t; s < kTS; s += blockDim.x) {
      int rel[4];
      rel_coords_fast(geo, gsx, min(tile * kTS + s, geo.V - 1), rel);
#pragma unroll
      for (int r = 0; r < 4; ++r) sm.zh[buf][s][r] = (double)coord_map_zerohalf(rel[r], geo.global[r]);
    }
  };
  if (t == 0) {
    mbar_init(&s_bar[0], 1);
    mbar_init(&s_bar[1], 1);
    fence_mbar_init();
    s_fail = 0;
  }
  __syncthreads();

  Neu acc_u[6][2], acc_s[4][2];
  double tu[6][2], ts[4][2];
#pragma unroll
  for (int k = 0; k < 6; ++k) tu[k][0] = tu[k][1] = 0.0;
#pragma unroll
  for (int s = 0; s < 4; ++s) ts[s][0] = ts[s][1] = 0.0;
  auto flush = [&]() {
#pragma unroll
    for (int k = 0; k < 6; ++k)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        acc_u[k][e].add(tu[k][e]);
        tu[k][e] = 0.0;
      }
#pragma unroll
    for (int s = 0; s < 4; ++s)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        acc_s[s][e].add(ts[s][e]);
        ts[s][e] = 0.0;
      }
  };

  long long const ntiles = (geo.V + kTS - 1) / kTS;
  long long tile = blockIdx.x;
  if (tile < ntiles) {
    if (t == 0) issue(tile, 0);
    zh_fill(tile, 0);
  }
  __syncthreads();
  int it = 0;
  bool more = false;
  for (; tile < ntiles; tile += gridDim.x, ++it) {
    int const st = it & 1;
    long long const s0 = tile * kTS;
    int const nvalid = (int)min((long long)kTS, geo.V - s0);
    more = tile + gridDim.x < ntiles;
    // the next tile into the other stage (its readers passed the last barrier)
    if (t == 0 && more) {
      fence_proxy_async_smem();
      issue(tile + gridDim.x, st ^ 1);
    }
    if (!mbar_wait(&s_bar[st], (uint32_t)((it >> 1) & 1))) s_fail = 1;
    else {
      const double* A_base = sm.stage[st][fl * 12 + ia];
      const double* B_base = sm.stage[st][NF * 12 + fl * 12 + ib];
      const double (*zhs)[4] = sm.zh[st];
      int z = (int)(s0 % geo.local[3]);
      int s = 0;
#pragma unroll 1
      while (s < nvalid) {
        // a run: sites of the tile with the same (t, x, y)
        int const end = min(nvalid, s + geo.local[3] - z), last = end - 1;
        // sums over the run, S of the products, T of zh_3 times them
        double S[4][2], T[4][2];
#pragma unroll
        for (int g = 0; g < 4; ++g) S[g][0] = S[g][1] = T[g][0] = T[g][1] = 0.0;
#pragma unroll 1
        for (; s < end; ++s) {
          const double2* A = reinterpret_cast<const double2*>(A_base + s * 24);
          const double2* B = reinterpret_cast<const double2*>(B_base + s * 24);
          // P[s1][s2] = sum_c conj(B[s1][c]) A[s2][c]: al = P02 - P31, be = P13 - P20,
          // ev = P03 + P21, od = P12 + P30
          double ar = 0, ai = 0, br = 0, bi = 0, er = 0, ei = 0, orr = 0, oi = 0;
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            double2 const y0 = B[c], y1 = B[3 + c], y2 = B[6 + c], y3 = B[9 + c];
            double2 const x0 = A[c], x1 = A[3 + c], x2 = A[6 + c], x3 = A[9 + c];
            ar += y0.x * x2.x; ar += y0.y * x2.y; ar -= y3.x * x1.x; ar -= y3.y * x1.y;
            ai += y0.x * x2.y; ai -= y0.y * x2.x; ai -= y3.x * x1.y; ai += y3.y * x1.x;
            br += y1.x * x3.x; br += y1.y * x3.y; br -= y2.x * x0.x; br -= y2.y * x0.y;
            bi += y1.x * x3.y; bi -= y1.y * x3.x; bi -= y2.x * x0.y; bi += y2.y * x0.x;
            er += y0.x * x3.x; er += y0.y * x3.y; er += y2.x * x1.x; er += y2.y * x1.y;
            ei += y0.x * x3.y; ei -= y0.y * x3.x; ei += y2.x * x1.y; ei -= y2.y * x1.x;
            orr += y1.x * x2.x; orr += y1.y * x2.y; orr += y3.x * x0.x; orr += y3.y * x0.y;
            oi += y1.x * x2.y; oi -= y1.y * x2.x; oi += y3.x * x0.y; oi -= y3.y * x0.x;
          }
          double const z3 = zhs[s][3];
          S[0][0] += ar; S[0][1] += ai; S[1][0] += br; S[1][1] += bi;
          S[2][0] += er; S[2][1] += ei; S[3][0] += orr; S[3][1] += oi;
          T[0][0] = fma(z3, ar, T[0][0]); T[0][1] = fma(z3, ai, T[0][1]);
          T[1][0] = fma(z3, br, T[1][0]); T[1][1] = fma(z3, bi, T[1][1]);
          T[2][0] = fma(z3, er, T[2][0]); T[2][1] = fma(z3, ei, T[2][1]);
          T[3][0] = fma(z3, orr, T[3][0]); T[3][1] = fma(z3, oi, T[3][1]);
        }
        z = 0;
        // X_0 = -(al + be), X_1 = -i (ev + od), X_2 = od - ev, X_3 = i (be - al)
        auto to_x = [](const double q[4][2], double x[4][2]) {
          x[0][0] = -(q[0][0] + q[1][0]); x[0][1] = -(q[0][1] + q[1][1]);
          x[1][0] = q[2][1] + q[3][1];    x[1][1] = -(q[2][0] + q[3][0]);
          x[2][0] = q[3][0] - q[2][0];    x[2][1] = q[3][1] - q[2][1];
          x[3][0] = q[0][1] - q[1][1];    x[3][1] = q[1][0] - q[0][0];
        };
        double X[4][2], W[4][2];
        to_x(S, X);
        to_x(T, W);
        const double* zh = zhs[last];
#pragma unroll
        for (int k = 0; k < 6; ++k) {
          int const r = comb_rho(k), g = comb_sigma(k);
#pragma unroll
          for (int e = 0; e < 2; ++e)
            tu[k][e] += g == 3 ? zh[r] * X[3][e] - W[r][e] : zh[r] * X[g][e] - zh[g] * X[r][e];
        }
#pragma unroll
        for (int g = 0; g < 4; ++g) { ts[g][0] += X[g][0]; ts[g][1] += X[g][1]; }
      }
      if ((it & (kFlushTiles - 1)) == kFlushTiles - 1) flush();
    }
    if (more) zh_fill(tile + gridDim.x, st ^ 1);
    __syncthreads();  // the stage and zh[st] are rewritten after this
    if (s_fail) break;
  }
  flush();
  if (s_fail) {
    // a wait gave up: report it, and let no copy into this CTA's shared
    // memory outlive it (bounded, as everything else)
    if (t == 0) {
      if (err) atomicExch(err, kErrWaitTimeout);
      mbar_wait(&s_bar[it & 1], (uint32_t)((it >> 1) & 1));
      if (more) mbar_wait(&s_bar[(it + 1) & 1], (uint32_t)(((it + 1) >> 1) & 1));
    }
    return;
  }
  double* out = partials + (((size_t)pi * gridDim.x + blockIdx.x) * NF + fl) * kDzLen;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    out[((k * 12 + ia) * 12 + ib) * 2] = acc_u[k][0].get();
    out[((k * 12 + ia) * 12 + ib) * 2 + 1] = acc_u[k][1].get();
  }
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    out[kDzuLen + ((s * 12 + ia) * 12 + ib) * 2] = acc_s[s][0].get();
    out[kDzuLen + ((s * 12 + ia) * 12 + ib) * 2 + 1] = acc_s[s][1].get();
  }
}

}  // namespace p1d

template <int NF>
static int p1f64_init_t(int nsm, int& grid) {
  size_t const smem = sizeof(p1d::Smem<NF>);
  cudaError_t e = cudaFuncSetAttribute(p1d::p1f64_kernel<NF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(p1d::p1f64_kernel<NF>, cudaFuncAttributePreferredSharedMemoryCarveout,
                             cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return cuda_fail(e, "p1f64 smem attribute");
  int nb = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, p1d::p1f64_kernel<NF>, NF * 144, smem);
  if (e != cudaSuccess) return cuda_fail(e, "p1f64 occupancy");
  if (nb < 1) return fail(HLBL_ECUDA, "p1f64 kernel cannot be resident (smem %zu)", smem);
  grid = nb * nsm;
  return HLBL_OK;
}

int p1f64_init(int nf, int nsm, int& grid) { return nf == 1 ? p1f64_init_t<1>(nsm, grid) : p1f64_init_t<2>(nsm, grid); }

long long p1f64_tiles(long long V) { return (V + p1d::kTS - 1) / p1d::kTS; }

void p1f64_launch(int nf, int grid, cudaStream_t st, const double* y, const PairBatch& b, const Geometry& geo,
                  int f0, double* partials, int* err) {
  if (nf == 2)
    p1d::p1f64_kernel<2><<<dim3(grid, b.n), 288, sizeof(p1d::Smem<2>), st>>>(y, b, geo, f0, partials, err);
  else
    p1d::p1f64_kernel<1><<<dim3(grid, b.n), 144, sizeof(p1d::Smem<1>), st>>>(y, b, geo, f0, partials, err);
}

}  // namespace hg
