// p1_f64.h -- the FP64 pass 1 (p1_f64.cu) as seen by the context code and the
// allocation-free entry.
#pragma once

#include <cuda_runtime.h>

#include "contract_kernels.cuh"

namespace hg {

// resident CTAs of the kernel for nf flavours on the current device
int p1f64_init(int nf, int nsm, int& grid);
long long p1f64_tiles(long long V);
// partials in p1_kernel's layout: [pair][cta][nf][kDzLen]
void p1f64_launch(int nf, int grid, cudaStream_t st, const double* y, const PairBatch& b, const Geometry& geo,
                  int f0, double* partials, int* err);

}  // namespace hg
