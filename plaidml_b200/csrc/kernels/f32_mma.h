// fp32 matrix products and convolutions on the bf16 tensor pipe, operands split on the way into shared memory.
#pragma once

#include <cuda_runtime.h>

#include <string>

#include "tc_launch.h"

namespace pmlb {

// Tile width (64, 128: one CTA; 256: a CTA pair), the number of CTAs (1..8) that share a tile's K range, and the estimated
// time.  bn 0: more tiles than a launch takes.
struct F32MmaTiles {
  int bn = 64, split = 1;
  double us = 0;
  bool one_order = false;   // the same additions in the same order whatever the width
};

// C[b][i][j] = sum_k A(b, i, k) * B(b, k, j), everything fp32 in device memory.
struct F32MmaLaunch {
  int m = 0, n = 0, k = 0, batch = 1;
  const float* a = nullptr;
  long long lda = 0, a_batch = 0;   // a_mn false: A(i, k) at a[i * lda + k]; true: at a[k * lda + i]
  bool a_mn = false;
  const ConvGeom* conv = nullptr;   // non-null: A is an NHWC activation at `a` (c a multiple of 4),
                                    // row i = output pixel i, k = (tap, channel); m, n, k, batch = n*p*q, k_out, r*s*c, 1
  const float* b = nullptr;
  long long ldb = 0, b_batch = 0;   // b_mn false: B(k, j) at b[j * ldb + k]; true: at b[k * ldb + j]
  bool b_mn = false;
  float* out = nullptr;             // may be null with row maxima
  long long ldc = 0, out_batch = 0;
  int epi_flags = 0;                // kEpi*; bias f32[n], residual f32 rows ldr apart
  const float* bias = nullptr;
  const float* residual = nullptr;
  long long ldr = 0, res_batch = 0;
  float* rowmax = nullptr;          // f32[batch * m], filled with -inf by the caller
  bool contraction = false;         // tiles without pairs; results that the parts cannot give are added again (f32_mma.cu)
  int* status = nullptr;            // device word that receives a non-zero code if a wait times out
  F32MmaTiles tiles;
};

// Whether the kernel accepts a convolution.
bool f32_mma_takes_conv(const ConvGeom& g);

struct F32MmaShape {
  int m = 0, n = 0, k = 0, batch = 1;
  bool conv = false;
  bool aligned_in = true, aligned_out = true;   // rows start on 16-byte boundaries
  long long elems = 0;                          // elements that each call's pre-pass would split
  int tile_n = 0;                               // 0 = choose; else 64 or 128
  bool whole_k = false;                         // one order of additions whatever the number of rows and tiles
  bool short_chains = false;                    // no CTA pairs, whose accumulator chains run over all of K
};

// The tiles a shape is expected to run fastest with.
F32MmaTiles f32_mma_tiles(const F32MmaShape& shape);

// Whether the kernel is expected to be faster than splitting the operands into TF32 parts by pre-passes, and its tiles.
bool f32_mma_faster(const F32MmaShape& shape, F32MmaTiles* tiles);

// A status word of the library's own on the current device, for plans that hold no device memory (so that they can be made
// and freed while a stream is being captured, and a captured graph outlive its plan); null if the device has none to give.
int* f32_mma_status_word();

// Returns 0 on success, otherwise a pmlb_status value with a message in *err.
int f32_mma_launch(const F32MmaLaunch& launch, cudaStream_t stream, std::string* err);

// Filter of an fp32 convolution as the kernel reads it: [taps][c][k] of f32, bf16 or f16 -> the same in f32.
cudaError_t launch_filter_to_f32(const void* in, int in_dtype, float* out, long long elems, cudaStream_t stream);

}  // namespace pmlb
