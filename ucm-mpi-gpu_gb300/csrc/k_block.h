// k_block.h -- block (Chebyshev-filtered subspace iteration) kernels.
#pragma once

#include <cuda_runtime.h>

#include "gpb_internal.h"
#include "k_eig.h"

namespace gpb {

constexpr int kBlk = 32;          // block width
constexpr int kMaxCheb = 128;     // largest filter degree

struct BlkArgs {
  const PatchDev* patches;
  const EigTile* tiles;
  const int* tile_begin;
  const int* tile_count;
  const float* a_up;
  const float* a_diag;
  long long lvec;
  const float3* coef;   // [npatch][max_steps] (alpha, beta, gamma)
  int max_steps;
  double* part;         // partial sums, FP32 hi + lo pairs: [ntiles * kBlkSplit][1 or 2 Gram
                        // matrices, or 32 residuals]
  int* counter;         // [npatch]
  const int* active;    // [npatch]
  const int* done;      // [npatch]
  const double* mat;    // [npatch][32*32]
  const double* theta;  // [npatch][32]
  int coarse;           // 0: fine radius-5 disk, 1: coarse 7 x 7 square
  const float* afull;   // stencil rows in the step's tile layout (k_block.cu): 84 floats
                        // (fine) / 52 (coarse) per pixel of a 16 x 16 tile
  int* err;             // set to 1 when a tile's staging wait gave up
};

// coarse level (2 x 2 aggregation)
constexpr int kCR = 3, kCW = 2 * kCR + 1, kCN = kCW * kCW;
struct CoarseArgs {
  const PatchDev* fine;
  const PatchDev* coarse;
  const int4* work;      // coarse 16 x 16 tiles
  const int4* work_f;    // fine 16 x 16 tiles
  const float* wsym_up;  // fine symmetric affinities (upper offsets)
  const float* deg;      // fine degrees
  long long lvec_f, lvec_c;
  float* wc;             // [coarse tiles][256][kCoarseNC]: A_c's rows in the step's tile layout
  float* degc;
  float* disc;
};
cudaError_t cf_launch_coarsen(const CoarseArgs& c, int nwork_c, cudaStream_t s);
cudaError_t cf_launch_full(const PatchDev* patches, const int4* work16, int nwork, const float* a_up,
                           const float* a_diag, long long lvec, float* afull, cudaStream_t s);
cudaError_t cf_launch_prolong(const CoarseArgs& c, int nwork_f, const float* xc, float* xf, cudaStream_t s);

void upload_block(const HostTables& t, cudaStream_t s);
// cf_step's tiles are those of the 16 x 16 work list, whose entries' .w is the
// tile's index in that list (the place of its coefficients)
constexpr int kStepTile = 16;
constexpr int kFullNC = 84, kCoarseNC = 52;      // floats per pixel's stencil row
constexpr int kBlkSplit = 4;  // CTAs per eigensolver tile in cf_gram / cf_rotate / cf_resid
// variant (bit-identical results, chosen by the autotuner): 0 computes 16 x 16
// pixels per CTA and pass, 1 halves them (for launches of few tiles)
constexpr int kStepVariants = 2, kStepDefault = 0;
// overlap: the launch before it on the stream is a step with the same active
// patches, tiles and operator, whose tail this one's set-up may overlap
cudaError_t cf_launch_step(const BlkArgs& a, const int4* work, int nwork, const float* Y, const float* X, float* out,
                           int step, cudaStream_t s, bool comp = false, int variant = kStepDefault,
                           bool overlap = false);
// out = U^T V per patch; with out2, out2 = U^T U in the same pass
cudaError_t cf_launch_gram(const BlkArgs& a, int npatch, int ntiles, const float* U, const float* V, double* out,
                           cudaStream_t s, double* out2 = nullptr);
cudaError_t cf_launch_rotate(const BlkArgs& a, int ntiles, float* U, float* V, int ncols, cudaStream_t s,
                             bool comp = false);
cudaError_t cf_launch_resid(const BlkArgs& a, int ntiles, const float* X, const float* AX, double* out,
                            cudaStream_t s);
cudaError_t cf_launch_extract(const BlkArgs& a, int ntiles, const float* X, float* evec, int nvec,
                              cudaStream_t s);
cudaError_t cf_launch_init(const BlkArgs& a, int ntiles, float* X, cudaStream_t s);

}  // namespace gpb
