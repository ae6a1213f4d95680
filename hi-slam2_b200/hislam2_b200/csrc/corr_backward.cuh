// Tiled gradients of the on-the-fly correlation (corr_backward.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace hs2 {

// The tile kernel covers 128 channels and radius <= 6 (142 KB of shared memory at 6).
constexpr int kCbMaxRadius = 6;

bool altcorr_bwd_tiled_ok(int b, int n1, int n2, int c, int m, int radius);
// workspace of a call of m edges, which pack the min(frames, m) frames that they can use on a side
size_t altcorr_bwd_tiled_bytes(int b, int n1, int n2, int h, int w, int h2, int w2, int m);
int altcorr_bwd_tiled(int dtype, const void* fmap1, const void* fmap2, int b, int n1, int n2, int h, int w, int h2,
                      int w2, const float* coords, const int64_t* ii, const int64_t* jj, int m, const float* grad,
                      int radius, float scale, void* g1, void* g2, int32_t* info, void* ws, cudaStream_t s);

}  // namespace hs2
