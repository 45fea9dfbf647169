// FP32 image <-> grid transforms in two fused passes (gb_fft.cu).
#pragma once

#include <cuda_runtime.h>

namespace gb {

// Whether the transforms below take size n: even, 16 .. 8192, no prime factor
// above 7.
bool fft_size_ok(int n);
// As gb_image_to_grid_f32 / gb_grid_to_image_f32 (taper may be NULL).
int fft_image_to_grid(const float* x, const float* taper, int n, float2* g, cudaStream_t s);
int fft_grid_to_image(const float2* g, const float* taper, int n, float2* w, float* x,
                      cudaStream_t s);

}  // namespace gb
