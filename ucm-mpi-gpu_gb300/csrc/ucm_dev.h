// ucm_dev.h -- device scratch and launchers of the OWT-UCM stages (k_ucm.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace gpb {

struct UcmImage {
  int H, W;
  long long pix;  // first pixel of the image in the per-pixel arrays
  int row0;       // first row in the per-row arrays
  long long wpix; // first cell in the flooding's labels, which have a border of one pixel
};

struct UcmScratch {
  unsigned* mm;        // complement of the ordered min, ordered max of pb
  float* pb;           // N
  uint8_t* q;          // N
  int32_t* off;        // H x 257
  uint16_t* cols;      // N
  UcmImage* img;       // this image's entry of the batch's image table
  int32_t* ws;         // all images' flooding labels, (H+2)(W+2) each
  uint8_t* bw;         // N
  float* wswt;         // N
  int32_t* paint_pix;  // painted pixels
  uint8_t* paint_ori;  // their orientation planes
  float* pb2;          // 4N
  int32_t* rowcnt;     // 2H
  int32_t* nart;       // 1
  int32_t* art;        // 4N at most
  int32_t* par;        // 4N
  int32_t* rank;       // 4N
  int32_t* bsum;       // 4N / 4096 + 1
  int32_t* nreg;       // 1
  int32_t* labels;     // N
  float* wswt2;        // (2H+1)(2W+1)
};

// The CTAs of a launch belong to the images one after the other, each with as
// many as its own size asks for: by pixels, by cells of the doubled grid, by
// rows, by painted pixels, by blocks of the scan.  (As many as the largest
// image for every one would be 36 M CTAs by rows for an image of 6000 x 2 among
// 6000 of 2 x 2, which have 18 K rows together.)
enum UcmKind { kUcmPix, kUcmCells, kUcmRows, kUcmPaint, kUcmScan, kUcmKinds };

// one image of a batch, as the kernels see it
struct UcmView {
  UcmScratch s;
  const float* orient;   // 8 planes
  int H, W, np;          // np: painted pixels
  int first[kUcmKinds];  // its first CTA in launches of each kind
};
// what sizes the launches of a batch
struct UcmBatch {
  const UcmView* views;  // device: n images, and an entry behind them whose `first` are the CTAs of all
  int n;
  int ctas[kUcmKinds];
  long long total_pix;
  long long ws_cells;    // of all images' flooding labels
};
// fills the `first` of n + 1 views and b.ctas
void ucm_ctas(UcmView* views, UcmBatch& b);

// max over orientations, quantisation, per-row level sort; base is image 0's
// view, whose arrays start the batch's concatenated ones
cudaError_t ucm_prepare(const UcmBatch& b, const UcmScratch& base, cudaStream_t st);
// flooding (one CTA per image) and the watershed-pixel map
cudaError_t ucm_flood(const UcmBatch& b, const UcmScratch& base, cudaStream_t st);
cudaError_t ucm_paint(const UcmBatch& b, const UcmScratch& base, cudaStream_t st);
cudaError_t ucm_mid(const UcmBatch& b, cudaStream_t st);

}  // namespace gpb
