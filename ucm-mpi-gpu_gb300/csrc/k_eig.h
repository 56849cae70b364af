// k_eig.h -- shared definitions of the eigensolver kernels.
#pragma once

#include <cuda_runtime.h>

#include "gpb_internal.h"

namespace gpb {

constexpr int kEigThreads = 256;
constexpr int kEigWarps = kEigThreads / 32;
constexpr int kEigPix = 8;                          // pixels per thread in the reductions
constexpr int kEigTile = kEigThreads * kEigPix;     // pixels per tile
constexpr int kMaxKrylov = 64;

struct EigTile {
  int patch, p0, p1, pad;
};

// everything the eigensolver kernels read, passed by value
struct EigArgs {
  const PatchDev* patches;
  const EigTile* tiles;
  const int* tile_begin;
  const int* tile_count;
  const float* a_up;     // 40 x lvec
  const float* a_diag;   // lvec
  float* V;              // (m+1) x lvec, current basis
  double* part;          // [ntiles * warps][m+1]
  double* hbuf;          // [npatch][m+1]
  double* T;             // [npatch][m*m]
  double* Y;             // [npatch][m*m]
  double* beta2;         // [npatch]
  int* counter;          // [npatch]
  const int* active;     // [npatch]
  const int* decision;   // [npatch]
  const int* nkeep;      // [npatch]
  long long lvec;
  int m, mp1;
};

void upload_eig(const HostTables& t, cudaStream_t s);
cudaError_t ks_launch_init(const EigArgs& a, int ntiles, float* w, cudaStream_t s);
// Batches of up to this many tiles take the five-launch step, which spreads a
// tile's work over several CTAs.  Milliseconds of one solve, three launches
// against five: 27.6 / 21.0 at 3 tiles, 124.1 / 96.4 at 22, 330.8 / 297.7 at
// 76, 434.1 / 427.8 at 88, 421.7 / 428.1 at 102, 573.6 / 617.9 at 118 and
// 739 / 782 at 560, where the extra reads of w and the launches cost more.
constexpr int kEigSplitTiles = 96;

// w = A v_j and h = V^T w
cudaError_t ks_launch_spmv(const EigArgs& a, int ntiles, int j, const float* src, int use_beta,
                           float* dst, cudaStream_t s);
// a Gram-Schmidt pass: mode 1 w -= V h, h2 = V^T w; mode 2 w -= V h2, |w|^2
cudaError_t ks_launch_orth(const EigArgs& a, int ntiles, int j, int mode, float* w, cudaStream_t s);
// the restart of the patches whose decision is 1 and the final Ritz vectors
// of those whose decision is 2 (each launched only when some patch needs it)
cudaError_t ks_launch_restart(const EigArgs& a, int ntiles, const float* w, float* vout, float* evec,
                              cudaStream_t s, bool any_restart, bool any_final);

}  // namespace gpb
