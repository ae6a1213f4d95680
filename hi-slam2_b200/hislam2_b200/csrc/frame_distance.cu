// frame_distance: per-edge mean optical-flow magnitude used for keyframe
// selection (reference: src/droid_kernels.cu:860-994, host side :2047-2069).
//
// One to eight warps per edge (enough to fill the GPU), each lane walking the edge's
// pixels; the sums are reduced with warp shuffles and, for several warps, one
// shared-memory pass.  HBM traffic is one disparity row per edge (4*ht*wd bytes, shared in
// L1 / L2 between the edges of a frame); the kernel is bound by instruction issue.
#include "common.cuh"
#include "profile.cuh"

namespace hs2 {

constexpr int kFdThreads = 256;

__device__ __forceinline__ float fd_rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float fd_sqrt(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Flow of a pixel at (a, b) = (u - cx, v - cy) from its projection's numerators:
//   du = (fx Y0 - a Y2) / Y2,  dv = (fy Y1 - b Y2) / Y2,
// which is fx Y0 / Y2 + cx - u without the difference of two image coordinates.  The point
// is Y = R [a/fx, b/fy, 1] + d t, so fx Y0, fy Y1 and Y2 are linear in (a, b, d); with the
// translation alone (R = 1) the numerators reduce to d (fx t0 - a t2) and d (fy t1 - b t2).
// One approximate reciprocal and square root per flow (relative error 2^-23, either sign).
// 90,000 pairs of 43x77 frames: 0.49 ms, against 1.76 ms for two projections with IEEE
// divisions per pixel; error against 64 bits 4.7e-8, before 5.6e-8.
template <int kWarps>   // warps per edge
__global__ void __launch_bounds__(kFdThreads)
frame_distance_kernel(const float* __restrict__ poses, int64_t num_poses, const float* __restrict__ disps,
                      int64_t num_disps, int ht, int wd, const float* __restrict__ intr,
                      const int64_t* __restrict__ ii, const int64_t* __restrict__ jj, int64_t num_edges, float beta,
                      float* __restrict__ dist, int32_t* __restrict__ info) {
  constexpr int kLanes = 32 * kWarps;
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t e = (int64_t)blockIdx.x * (8 / kWarps) + wid / kWarps;
  float s1 = 0.f, s2 = 0.f;
  int n1 = 0, n2 = 0;
  bool ok = false;
  if (e < num_edges) {
    const int64_t ix = ii[e], jx = jj[e];
    ok = ix >= 0 && jx >= 0 && ix < num_poses && jx < num_poses && ix < num_disps;
    if (ok) {
      const float fx = intr[0], fy = intr[1], cx = intr[2], cy = intr[3];
      float t[3], q[4];
      relative_pose(poses + 7 * ix, poses + 7 * ix + 3, poses + 7 * jx, poses + 7 * jx + 3, t, q);
      const float x = q[0], y = q[1], z = q[2], w = q[3], ifx = 1.f / fx, ify = 1.f / fy;
      // Y2 = P + C2 with P = A2 a + B2 b + D2 d; the numerators take C2 out of Y2, so that the
      // diagonals of R enter as differences (R00 - R22, R11 - R22), formed without cancellation:
      // fx Y0 - a Y2 = A0 a + B0 b + C0 + D0 d - a P,  fy Y1 - b Y2 = A1 a + .. - b P
      const float A0 = 2.f * (x - z) * (x + z), B0 = 2.f * (x * y - z * w) * (fx * ify), C0 = 2.f * (x * z + y * w) * fx;
      const float A1 = 2.f * (x * y + z * w) * (fy * ifx), B1 = 2.f * (y - z) * (y + z), C1 = 2.f * (y * z - x * w) * fy;
      const float A2 = 2.f * (x * z - y * w) * ifx, B2 = 2.f * (y * z + x * w) * ify, C2 = 1.f - 2.f * (x * x + y * y);
      const float D0 = fx * t[0], D1 = fy * t[1], D2 = t[2];
      const int HW = ht * wd;
      const float* row = disps + ix * HW;
      int k = (wid % kWarps) * 32 + lane;
      const int du = kLanes % wd;
      const float dv = (float)(kLanes / wd);
      int u = k % wd;
      float b = (float)(k / wd) - cy;
#pragma unroll 4
      for (; k < HW; k += kLanes) {
        const float d = __ldg(row + k);
        const float a = (float)u - cx;
        const float P = fmaf(A2, a, fmaf(B2, b, D2 * d)), Y2 = P + C2;
        const float N0 = fmaf(-a, P, fmaf(A0, a, fmaf(B0, b, fmaf(D0, d, C0))));
        const float N1 = fmaf(-b, P, fmaf(A1, a, fmaf(B1, b, fmaf(D1, d, C1))));
        const float iy = fd_rcp(Y2), f0 = N0 * iy, f1 = N1 * iy;
        const float r1 = fd_sqrt(fmaf(f0, f0, f1 * f1));
        if (Y2 > kMinDepth) {
          s1 += r1;
          ++n1;
        }
        const float Z2 = fmaf(D2, d, 1.f), iz = d * fd_rcp(Z2);
        const float g0 = fmaf(-a, D2, D0) * iz, g1 = fmaf(-b, D2, D1) * iz;
        const float r2 = fd_sqrt(fmaf(g0, g0, g1 * g1));
        if (Z2 > kMinDepth) {
          s2 += r2;
          ++n2;
        }
        u += du;
        b += dv;
        if (u >= wd) {
          u -= wd;
          b += 1.f;
        }
      }
    }
  }
  // the lanes' sums and the final quotient in double: the result then carries little more than
  // the lanes' own rounding
  double d1 = s1, d2 = s2;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    d1 += __shfl_xor_sync(0xffffffffu, d1, o);
    d2 += __shfl_xor_sync(0xffffffffu, d2, o);
  }
  n1 = __reduce_add_sync(0xffffffffu, n1);
  n2 = __reduce_add_sync(0xffffffffu, n2);
  if (kWarps > 1) {
    __shared__ double fs[2][8];
    __shared__ int ns[2][8];
    if (lane == 0) {
      fs[0][wid] = d1;
      fs[1][wid] = d2;
      ns[0][wid] = n1;
      ns[1][wid] = n2;
    }
    __syncthreads();
    if (wid % kWarps) return;
    d1 = d2 = 0.0;
    n1 = n2 = 0;
    for (int g = 0; g < kWarps; ++g) {
      d1 += fs[0][wid + g];
      d2 += fs[1][wid + g];
      n1 += ns[0][wid + g];
      n2 += ns[1][wid + g];
    }
  }
  if (lane != 0 || e >= num_edges) return;
  if (!ok) {
    dist[e] = 1000.0f;
    if (info) atomicOr(info, HS2_DEV_BAD_INDEX);
    return;
  }
  const double db = beta, nb = 1.0f - beta;
  const double val = db * n1 + nb * n2, tot = (db + nb) * (double)(ht * wd);
  dist[e] = ((float)val / ((float)tot + 1e-8f) < 0.75f) ? 1000.0f : (float)((db * d1 + nb * d2) / val);
}

template <int kWarps>
static void fd_launch(const float* poses, int64_t num_poses, const float* disps, int64_t num_disps, int ht, int wd,
                      const float* intr, const int64_t* ii, const int64_t* jj, int64_t num_edges, float beta,
                      float* dist, int32_t* info, cudaStream_t s) {
  constexpr int kEdges = 8 / kWarps;   // edges per CTA
  frame_distance_kernel<kWarps><<<(unsigned)((num_edges + kEdges - 1) / kEdges), kFdThreads, 0, s>>>(
      poses, num_poses, disps, num_disps, ht, wd, intr, ii, jj, num_edges, beta, dist, info);
}

}  // namespace hs2

extern "C" int hs2_frame_distance(const float* poses, int64_t num_poses, const float* disps,
                                  int64_t num_disps, int ht, int wd, const float* intrinsics,
                                  const int64_t* ii, const int64_t* jj, int64_t num_edges, float beta,
                                  float* dist, int32_t* info, hs2_stream_t stream) {
  using namespace hs2;
  if (num_edges < 0 || ht <= 0 || wd <= 0 || num_poses < 0 || num_disps < 0) {
    set_error("frame_distance: bad sizes (edges=%lld ht=%d wd=%d)", (long long)num_edges, ht, wd);
    return HS2_ERR_INVALID;
  }
  if (num_edges == 0) return HS2_OK;
  if (num_edges > 0x7fffffff) {
    set_error("frame_distance: too many edges");
    return HS2_ERR_INVALID;
  }
  int rc = bind_device(dist);
  if (rc) return rc;
  HS2_PROF("frame_distance", (cudaStream_t)stream);
  // A warp per edge once that fills the GPU; more for fewer edges, whose time is the walk of one
  // edge's pixels.  43x77, one / four / eight warps per edge: 600 edges 12.9 / 8.2 / 7.8 us,
  // 1184: 13.1 / 10.2 / 11.4, 1800: 17.2 / 15.6 / 16.7, 2368: 17.2 / 17.7 / 20.4, 8000: 48.6 / 53.0 / 62.6.
  auto launch = num_edges >= 16 * kNumSMs ? fd_launch<1> : num_edges >= 8 * kNumSMs ? fd_launch<4> : fd_launch<8>;
  launch(poses, num_poses, disps, num_disps, ht, wd, intrinsics, ii, jj, num_edges, beta, dist, info,
         (cudaStream_t)stream);
  HS2_LAUNCH_CHECK("frame_distance_kernel");
  return HS2_OK;
}
