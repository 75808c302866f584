// p2_f64.h -- the FP64 pass 2 (p2_f64.cu) as seen by the context code.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

#include "contract_kernels.cuh"

namespace hg {

// resident CTAs for one ([0]) and two ([1]) flavours
int p2f64_init(int nsm, int grid[2]);
// doubles of dzq per (pair, flavour)
size_t p2f64_dzq_len();
long long p2f64_tiles(long long V);
// dzq from pass 1's sums dz, or (dz null, one pair and flavour) from sums with
// the gammas inserted; *bad is set where those are not four images of one dz
void p2f64_launch_dzq(const double* dz, const double* g_dzu, const double* g_dzsu, int nf, int npairs, double* dzq,
                      int* bad, cudaStream_t st);
// skip: the kernel does nothing where *skip is set (null: never)
void p2f64_launch(int nf, int grid, cudaStream_t st, const double* y, const PairBatch& b, const Geometry& geo,
                  const P2Args& a, const double* dzq, double* partials, int* err, const int* skip);

}  // namespace hg
