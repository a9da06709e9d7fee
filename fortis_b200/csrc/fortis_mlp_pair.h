// Interface of the fp32 MLP layers on pairs of CTAs (fortis_mlp_pair.cu)
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <string>

#include "fortis_plan.h"

namespace fortis {

// One layer: split activations [2][nrows][K padded to 32] times split weights, maps of boxes 32 x 64 and 32 x 128 rows
struct PairLayer {
  const float* a; long long nrows; int K, N;
  const CUtensorMap* map_hi[2]; const CUtensorMap* map_lo[2];
  const float* bias; int act; float slope;
  float* out;                                        // split output [2][nrows][N padded to 32], or ...
  float* Y;                                          // ... row-major [nrows][N], or ...
  const Access* store_by_slot; ArrayTable TS; long long cout[2][3]; RowGeom g;    // ... scattered (N <= 256)
  const float *out_mul, *relu_mask;
  double* partials; double* sum; unsigned int* done;
  int* status;
};
bool pair_available();                               // the kernels' shared memory and register splits are to be had
bool pair_wide(long long nrows, int N, bool scatter);      // tiles of 256 features, not 128
bool pair_layer(const PairLayer& L, cudaStream_t s, std::string* err);
void pair_split_gathered(const Access* slots, const ArrayTable& T, const RowGeom& g, int n_in, const float* in_div, float* out, long long nrows, cudaStream_t s);
void pair_split_rows(const float* X, int n_in, const float* in_div, float* out, long long nrows, cudaStream_t s);

}  // namespace fortis
