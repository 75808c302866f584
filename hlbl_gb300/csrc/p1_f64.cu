// p1_f64.cu -- the FP64 pass 1 (ker_dzu_dzsu, cuda_lattice.cu:160-262) with its
// products in 64-bit integers.
//
// Thread (ia, ib) of flavour f = f0 + blockIdx.z owns dzu[k][ia][ib] and
// dzsu[s][ia][ib], as in p1_kernel. The FP64 pipe gives two multiply-adds per SM
// and cycle here, the integer multiply-add (32 x 32 + 64 bits) 64: a tile's rows
// are turned into integers of 55 bits and a sign below the row's largest value
// (an exponent per row and tile of 8 sites), held as two limbs of 28 bits, and a
// product takes three integer multiply-adds (the low limbs' product, below 2^-54
// of the largest product, is dropped; no other rounding until a site's sum of 12
// products is put together). As the zerohalf weights zh_0..zh_2 are constant along a
// run of sites in z and zh_3 grows by one from site to site, a run needs the sum S
// of its products and the sum W of S's partial sums, both exact in 64 bits; FP64
// takes over at the end of the run: the ten results from S and T = sum zh_3 x
// product = zh_3(first) S + (n S - W), those into the compensated sums every
// kFlushTiles tiles. Measured (both flavours, one pair): with FP64 products 42 ms
// at 663,552 sites and 0.54 ms at 8,192, so 13.4 and 0.24 (with two stages and three
// CTAs per SM 16.7 and 0.25: the CTAs hide each other's copies and barriers).
#include <cuda_runtime.h>

#include <cstdint>

#include "contract_kernels.cuh"
#include "hlbl_gb300.h"
#include "hlbl_internal.h"
#include "fixed_point.cuh"
#include "p1_f64.h"

namespace hg {
namespace p1d {

constexpr int kTS = 8;                 // sites per tile
constexpr int kRow = kTS * 24 + 2;     // staged row: 16 bytes of padding against bank conflicts
constexpr int kFlushTiles = 4;         // tiles per addition into the compensated sums
constexpr int kThreads = 144;
struct __align__(128) Smem {
  double stage[24][kRow];           // rows [src | y][12]; a tile at work holds limbs (hi, lo) instead
  int zh[2][kTS][4];
  int em[24];                          // the rows' exponents (exp_of)
};

__global__ void __launch_bounds__(kThreads, 4)
p1f64_kernel(const double* __restrict__ y, PairBatch batch, Geometry geo, int f0, double* __restrict__ partials,
             int* __restrict__ err) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
  __shared__ __align__(8) uint64_t s_bar;
  __shared__ int s_fail;
  int const t = threadIdx.x, pi = blockIdx.y, fl = blockIdx.z, nf = gridDim.z;
  const double* __restrict__ src = batch.p[pi].src;
  int const gsx[4] = {batch.p[pi].gsx[0], batch.p[pi].gsx[1], batch.p[pi].gsx[2], batch.p[pi].gsx[3]};
  int const ia = t / 12, ib = t % 12;
  // src flavour f0 + fl, y flavour 1 - (f0 + fl)
  auto issue = [&](long long tile) {
    long long const s0 = tile * kTS;
    uint32_t const bytes = (uint32_t)min((long long)kTS, geo.V - s0) * 192u;
    mbar_arrive_expect_tx(&s_bar, bytes * 24);
    for (int row = 0; row < 24; ++row) {
      int const i = row % 12, ff = row < 12 ? f0 + fl : 1 - f0 - fl;
      bulk_g2s(sm.stage[row], (row < 12 ? src : y) + ((size_t)(ff * 12 + i) * geo.V + s0) * 24, bytes, &s_bar);
    }
  };
  auto zh_fill = [&](long long tile, int buf) {
    for (int s = t; s < kTS; s += kThreads) {
      int rel[4];
      rel_coords_fast(geo, gsx, min(tile * kTS + s, geo.V - 1), rel);
#pragma unroll
      for (int r = 0; r < 4; ++r) sm.zh[buf][s][r] = coord_map_zerohalf(rel[r], geo.global[r]);
    }
  };
  if (t == 0) {
    mbar_init(&s_bar, 1);
    fence_mbar_init();
    s_fail = 0;
  }
  if (t < 24) sm.em[t] = kZeroExp;
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
    if (t == 0) issue(tile);
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
    if (!mbar_wait(&s_bar, (uint32_t)(it & 1))) s_fail = 1;
    __syncthreads();
    if (s_fail) break;
    {
      // the rows' exponents, then limbs in place: six threads per row
      int const row = t / 6, nval = nvalid * 24;
      double* const p = sm.stage[row];
      int m = kZeroExp;
#pragma unroll 8
      for (int i = t % 6; i < nval; i += 6) m = max(m, exp_of(p[i], 0));
      atomicMax(&sm.em[row], m);
      __syncthreads();
      m = sm.em[row];
#pragma unroll 4
      for (int i = t % 6; i < nval; i += 6) {
        long long const x = to_fixed<2>(p[i], 0, m);  // |x| <= 2^55
        int const hi = (int)((x + (1ll << 27)) >> 28), lo = (int)(x - ((long long)hi << 28));
        *reinterpret_cast<int2*>(p + i) = make_int2(hi, lo);
      }
    }
    __syncthreads();
    {
      const double* A_base = sm.stage[ia];
      const double* B_base = sm.stage[12 + ib];
      const int (*zhs)[4] = sm.zh[st];
      // a product's unit 2^56 2^(em - 1077) 2^(em' - 1077)
      int const ea = sm.em[ia], eb = sm.em[12 + ib];
      double const scale = ea == kNoScale || eb == kNoScale ? __longlong_as_double(0x7FF8000000000000ll)
                                                            : pow2(ea + eb - 2 * 1077 + 56);
      int z = (int)(s0 % geo.local[3]);
      int s = 0;
#pragma unroll 1
      while (s < nvalid) {
        // a run: sites of the tile with the same (t, x, y) and zh_3 growing by one
        int const first = s;
        long long S[8], W[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) S[i] = W[i] = 0;
#pragma unroll 1
        do {
          const int4* A = reinterpret_cast<const int4*>(A_base + s * 24);
          const int4* B = reinterpret_cast<const int4*>(B_base + s * 24);
          // P[s1][s2] = sum_c conj(B[s1][c]) A[s2][c]: al = P02 - P31, be = P13 - P20,
          // ev = P03 + P21, od = P12 + P30; each as hi.hi and hi.lo + lo.hi
          long long h[8], m[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) h[i] = m[i] = 0;
          auto mac = [&](int i, int ah, int al, int bh, int bl) {
            h[i] += (long long)ah * bh;
            m[i] += (long long)ah * bl;
            m[i] += (long long)al * bh;
          };
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            int4 const y0 = B[c], y1 = B[3 + c], y2 = B[6 + c], y3 = B[9 + c];
            {
              int4 const x2 = A[6 + c];
              mac(0, y0.x, y0.y, x2.x, x2.y); mac(0, y0.z, y0.w, x2.z, x2.w);
              mac(1, y0.x, y0.y, x2.z, x2.w); mac(1, -y0.z, -y0.w, x2.x, x2.y);
              mac(6, y1.x, y1.y, x2.x, x2.y); mac(6, y1.z, y1.w, x2.z, x2.w);
              mac(7, y1.x, y1.y, x2.z, x2.w); mac(7, -y1.z, -y1.w, x2.x, x2.y);
            }
            {
              int4 const x3 = A[9 + c];
              mac(2, y1.x, y1.y, x3.x, x3.y); mac(2, y1.z, y1.w, x3.z, x3.w);
              mac(3, y1.x, y1.y, x3.z, x3.w); mac(3, -y1.z, -y1.w, x3.x, x3.y);
              mac(4, y0.x, y0.y, x3.x, x3.y); mac(4, y0.z, y0.w, x3.z, x3.w);
              mac(5, y0.x, y0.y, x3.z, x3.w); mac(5, -y0.z, -y0.w, x3.x, x3.y);
            }
            {
              int4 const x1 = A[3 + c];
              mac(0, -y3.x, -y3.y, x1.x, x1.y); mac(0, -y3.z, -y3.w, x1.z, x1.w);
              mac(1, -y3.x, -y3.y, x1.z, x1.w); mac(1, y3.z, y3.w, x1.x, x1.y);
              mac(4, y2.x, y2.y, x1.x, x1.y); mac(4, y2.z, y2.w, x1.z, x1.w);
              mac(5, y2.x, y2.y, x1.z, x1.w); mac(5, -y2.z, -y2.w, x1.x, x1.y);
            }
            {
              int4 const x0 = A[c];
              mac(2, -y2.x, -y2.y, x0.x, x0.y); mac(2, -y2.z, -y2.w, x0.z, x0.w);
              mac(3, -y2.x, -y2.y, x0.z, x0.w); mac(3, y2.z, y2.w, x0.x, x0.y);
              mac(6, y3.x, y3.y, x0.x, x0.y); mac(6, y3.z, y3.w, x0.z, x0.w);
              mac(7, y3.x, y3.y, x0.z, x0.w); mac(7, -y3.z, -y3.w, x0.x, x0.y);
            }
          }
          // a site's sum stays below 2^57.6 units, eight sites' S and W below 2^63
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            S[i] += h[i] + ((m[i] + (1ll << 27)) >> 28);
            W[i] += S[i];
          }
          ++s;
          ++z;
        } while (s < nvalid && z < geo.local[3] && zhs[s][3] == zhs[s - 1][3] + 1);
        if (z == geo.local[3]) z = 0;
        double Q[4][2], R[4][2];  // al, be, ev, od: S and T
        {
          int const n = s - first;
          double const z0 = (double)zhs[first][3];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            Q[i >> 1][i & 1] = (double)S[i];
            R[i >> 1][i & 1] = fma(z0, Q[i >> 1][i & 1], (double)(n * S[i] - W[i]));
          }
        }
        // X_0 = -(al + be), X_1 = -i (ev + od), X_2 = od - ev, X_3 = i (be - al)
        auto to_x = [](const double q[4][2], double x[4][2]) {
          x[0][0] = -(q[0][0] + q[1][0]); x[0][1] = -(q[0][1] + q[1][1]);
          x[1][0] = q[2][1] + q[3][1];    x[1][1] = -(q[2][0] + q[3][0]);
          x[2][0] = q[3][0] - q[2][0];    x[2][1] = q[3][1] - q[2][1];
          x[3][0] = q[0][1] - q[1][1];    x[3][1] = q[1][0] - q[0][0];
        };
        double X[4][2];
        double Y[4][2];
        to_x(Q, X);
        to_x(R, Y);
        double const zh[3] = {(double)zhs[first][0], (double)zhs[first][1], (double)zhs[first][2]};
#pragma unroll
        for (int k = 0; k < 6; ++k) {
          int const r = comb_rho(k), g = comb_sigma(k);
#pragma unroll
          for (int e = 0; e < 2; ++e)
            tu[k][e] = fma(scale, g == 3 ? zh[r] * X[3][e] - Y[r][e] : zh[r] * X[g][e] - zh[g] * X[r][e], tu[k][e]);
        }
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          ts[g][0] = fma(scale, X[g][0], ts[g][0]);
          ts[g][1] = fma(scale, X[g][1], ts[g][1]);
        }
      }
      if ((it & (kFlushTiles - 1)) == kFlushTiles - 1) flush();
    }
    if (more) zh_fill(tile + gridDim.x, st ^ 1);
    __syncthreads();  // the stage, zh[st] and em are rewritten after this
    // (one stage: the CTAs of an SM hide each other's copies)
    if (t == 0 && more) {
      fence_proxy_async_smem();
      issue(tile + gridDim.x);
    }
    if (t < 24) sm.em[t] = kZeroExp;
  }
  flush();
  if (s_fail) {
    // a wait gave up: report it, and let no copy into this CTA's shared
    // memory outlive it (bounded, as everything else)
    if (t == 0) {
      if (err) atomicExch(err, kErrWaitTimeout);
      mbar_wait(&s_bar, (uint32_t)(it & 1));
    }
    return;
  }
  double* out = partials + (((size_t)pi * gridDim.x + blockIdx.x) * nf + fl) * kDzLen;
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

int p1f64_init(int nf, int nsm, int& grid) {
  size_t const smem = sizeof(p1d::Smem);
  cudaError_t e = cudaFuncSetAttribute(p1d::p1f64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(p1d::p1f64_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return cuda_fail(e, "p1f64 smem attribute");
  int nb = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, p1d::p1f64_kernel, p1d::kThreads, smem);
  if (e != cudaSuccess) return cuda_fail(e, "p1f64 occupancy");
  if (nb < 1) return fail(HLBL_ECUDA, "p1f64 kernel cannot be resident (smem %zu)", smem);
  grid = nb * nsm / nf;
  return HLBL_OK;
}

long long p1f64_tiles(long long V) { return (V + p1d::kTS - 1) / p1d::kTS; }

void p1f64_launch(int nf, int grid, cudaStream_t st, const double* y, const PairBatch& b, const Geometry& geo,
                  int f0, double* partials, int* err) {
  p1d::p1f64_kernel<<<dim3(grid, b.n, nf), p1d::kThreads, sizeof(p1d::Smem), st>>>(y, b, geo, f0, partials, err);
}

}  // namespace hg
