// p2_dig.h -- the FP64 pass 2 by digit products (p2_dig.cu) as seen by the
// context code.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

#include "contract_kernels.cuh"

namespace hg {

int p2dig_init();
// Bytes of the work buffer for lattices of up to V sites (bounded: larger
// lattices are taken in batches of sites).
size_t p2dig_ws_bytes(long long V, int nsm);
// Pass 2 of one pair (its source, gsx and yv in wa.batch.p[0]; a.w and a.coef null:
// the exact weight is evaluated on the way), from pass 1's sums dz or
// from sums with the gammas inserted (dz null); partials[cta*nf + fl], nsm CTAs.
void p2dig_launch(int nf, int nsm, cudaStream_t st, const double* y, const WArgs& wa, const QedF32& qf, const Geometry& geo,
                  const P2Args& a, const double* dz, const double* g_dzu, const double* g_dzsu, void* ws,
                  double* partials, int* err);

}  // namespace hg
