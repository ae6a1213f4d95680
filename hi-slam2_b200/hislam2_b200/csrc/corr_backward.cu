// Gradients of the on-the-fly correlation by 8x8 pixel tiles (128 channels).
//
// Backward of one edge at one level: with G[p][t] the adjoint of the bilinear blend (the
// gradient of the inner product of pixel p's features and target position t),
//   g1[p] = sum_t G[p][t] f2[t],     g2[t] += sum_p G[p][t] f1[p].
// Both are 128-long axpys; a pixel-by-pixel kernel re-reads f2 for every pixel and sends
// every (pixel, tap) product to memory as an atomic.  Here a CTA owns an 8x8 tile, as 16
// groups of 2x2 pixels:
//   * features and gradients are channel-last in FP32 (corr_bwd_pack; only frames that an edge
//     uses have a place, so the workspace follows the edges), so one position is one 512-byte row
//     and a warp holds it as one float4 per lane;
//   * the window gradients of a group are laid out over the union of its four windows, one
//     float4 (four pixels) per position, so one shared-memory broadcast feeds 16 FMAs;
//   * g1: one warp per group walks the union, reading each f2 row once for four pixels;
//   * g2: one warp per 2x2 block of positions gathers the groups that reach it (64 FMAs
//     per four f1 rows) and issues one vector reduction per position and tile, instead of
//     one atomic per pixel, tap and channel.
// All arithmetic is FP32 as in the pixel-by-pixel kernel.  Where a group's union does not
// fit its slot, or any feature is not finite (0 * inf would leak into pixels whose window
// does not hold it), the group keeps four separate windows and touches only those.
//
// Bound by shared-memory wavefronts and FMA issue together: a union position costs 5
// wavefronts and 16 FMAs (4 cycles of issue) per group.  Measured (84 edges, 48x64, radius
// 4, four levels, B200): 2.50 ms for the tiles plus 0.16 / 0.12 ms to pack (and pool) / unpack,
// against 27.3 ms for the pixel-by-pixel kernel (altcorr_bwd_kernel, kept for other
// channel counts and radius > 6).  Packing and unpacking move 530 and 400 MB there (81 and
// 61 us at the copy rate); with index arithmetic and one load in flight per element they took
// 192 and 343 us, by warp-owned rows with eight to sixteen loads in flight 102 and 124.
#include <algorithm>

#include "common.cuh"
#include "profile.cuh"
#include "corr_backward.cuh"

namespace hs2 {

namespace {

constexpr int kCbC = 128;
constexpr int kCbThreads = 512;      // 16 warps = 16 groups of 2x2 pixels
constexpr int kCbPackPix = 64;       // pixels of a transposed block
constexpr int kCbPackCh = 256 / kCbPackPix;   // channels that its 256 threads hold at once

struct CbArgs {
  const float* f1;                   // [B*S1][H*W][128]
  const float* f2[4];                // [B*S2][H2*W2][128] per level
  float* o1;
  float* o2[4];
  const float* coords;               // [B][M][2][H][W], or [B][M][H][W][2] when interleaved
  const void* grad;                  // [B][M][levels][2r+1 (x)][2r+1 (y)][H][W]
  const int64_t* ii;                 // null: frame m on both sides
  const int64_t* jj;
  const int* slot1;                  // with ii: where a frame's packed features and accumulator are
  const int* slot2;
  int N1, N2, S1, S2;                // frames, and packed frames a batch entry
  int M, H, W, r, levels, cap, interleaved;
  int H2[4], W2[4];
  float scale;
  const int32_t* nonfinite;
  int32_t* info;
};

struct CbGroup {
  int x0, y0, w, h;                  // union of the windows inside the target
  int mode;                          // 0 nothing, 1 union, 2 four windows
};

__device__ __forceinline__ void red4(float* p, const float4 v) {
  asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z),
               "f"(v.w)
               : "memory");
}
__device__ __forceinline__ void fma4(float4& a, const float g, const float4 v) {
  a.x = fmaf(g, v.x, a.x);
  a.y = fmaf(g, v.y, a.y);
  a.z = fmaf(g, v.z, a.z);
  a.w = fmaf(g, v.w, a.w);
}

// floats of the staged gradients (odd row length: consecutive taps hit consecutive banks);
// the f1 rows of the tile take the same bytes once the windows are formed
__host__ __device__ inline int cb_gstride(int r) {
  const int rd = 2 * r + 1;
  return (rd * rd) | 1;
}
inline size_t cb_stage_bytes(int r) {
  const size_t a = (size_t)64 * cb_gstride(r) * 4, b = (size_t)64 * kCbC * 4;
  return ((a > b ? a : b) + 15) & ~(size_t)15;
}
// positions a group's slot holds: the union of four windows spread by up to 6 pixels
inline int cb_cap(int r) { return (2 * r + 8) * (2 * r + 8); }
inline size_t cb_smem(int r) { return cb_stage_bytes(r) + (size_t)16 * cb_cap(r) * 16; }

// red1: several edges may share a source frame (g1 by reduction); otherwise a pixel of g1
// belongs to one CTA, which stores it at the first level and adds at the others.
// 64 registers: two CTAs per SM at radius <= 4 (98 KB of shared memory each).
template <typename TG, bool kRed1>
__global__ void __launch_bounds__(kCbThreads, 2) corr_bwd_tile_kernel(const __grid_constant__ CbArgs A) {
  extern __shared__ __align__(16) uint8_t cb_raw[];
  const int r = A.r, D = 2 * r + 2, rd = 2 * r + 1, H = A.H, W = A.W, HW = H * W;
  const int gst = cb_gstride(r);
  float* gs = reinterpret_cast<float*>(cb_raw);                    // [64][gst]
  float4* F1 = reinterpret_cast<float4*>(cb_raw);                  // [64][32], after gs
  const size_t stage = (((size_t)64 * max(gst, kCbC) * 4) + 15) & ~(size_t)15;
  float4* Gu = reinterpret_cast<float4*>(cb_raw + stage);          // [16][cap]
  __shared__ float4 geo[64];                                       // dx, dy, window x0, y0 (ints)
  __shared__ CbGroup grp[16];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int b = blockIdx.z, m = blockIdx.y;
  const int ntx = (W + 7) / 8;
  const int tx0 = ((int)blockIdx.x % ntx) * 8, ty0 = ((int)blockIdx.x / ntx) * 8;
  const int64_t ix = A.ii ? A.ii[m] : m, jx = A.jj ? A.jj[m] : m;
  if (!(ix >= 0 && ix < A.N1 && jx >= 0 && jx < A.N2)) {
    if (tid == 0 && blockIdx.x == 0 && A.info) atomicOr(A.info, HS2_DEV_BAD_INDEX);
    return;
  }
  const int64_t bm = (int64_t)b * A.M + m;
  const bool separate = *A.nonfinite != 0;
  const int gx = 2 * (warp & 3), gy = 2 * (warp >> 2);             // the warp's group inside the tile
  const int64_t fr1 = (int64_t)b * A.S1 + (A.ii ? A.slot1[ix] : m), fr2 = (int64_t)b * A.S2 + (A.ii ? A.slot2[jx] : m);
  const float4* f1 = reinterpret_cast<const float4*>(A.f1) + fr1 * HW * 32;
  float4* o1 = reinterpret_cast<float4*>(A.o1) + fr1 * HW * 32;

  for (int lvl = 0; lvl < A.levels; ++lvl) {
    const int H2 = A.H2[lvl], W2 = A.W2[lvl];
    const float4* f2 = reinterpret_cast<const float4*>(A.f2[lvl]) + fr2 * H2 * W2 * 32;
    float* o2 = A.o2[lvl] + fr2 * H2 * W2 * kCbC;
    __syncthreads();                                               // the previous level's F1 / Gu readers
    if (tid < 64) {
      const int px = tx0 + (tid & 7), py = ty0 + (tid >> 3);
      float4 g = make_float4(0.f, 0.f, __int_as_float(W2), __int_as_float(H2));   // outside the image: no taps
      if (px < W && py < H) {
        const int64_t p = (int64_t)py * W + px;
        const float s = 1.0f / (float)(1 << lvl);
        const float x = s * (A.interleaved ? A.coords[(bm * HW + p) * 2] : A.coords[bm * 2 * HW + p]);
        const float y = s * (A.interleaved ? A.coords[(bm * HW + p) * 2 + 1] : A.coords[(bm * 2 + 1) * HW + p]);
        const float fx = floorf(x), fy = floorf(y);
        // a window that starts at W2 or ends at 0 has no taps: clamping keeps the sums in range
        const int xw = min(max((int)fx, -2 * D), W2 + 2 * D) - r, yw = min(max((int)fy, -2 * D), H2 + 2 * D) - r;
        g = make_float4(x - fx, y - fy, __int_as_float(xw), __int_as_float(yw));
      }
      geo[tid] = g;
    }
    const TG* gr = static_cast<const TG*>(A.grad) + (bm * A.levels + lvl) * rd * rd * (int64_t)HW;
    for (int idx = tid; idx < 64 * rd * rd; idx += kCbThreads) {
      const int q = idx & 63, o = idx >> 6;
      const int px = tx0 + (q & 7), py = ty0 + (q >> 3);
      gs[q * gst + o] = (px < W && py < H) ? A.scale * to_f(gr[(int64_t)o * HW + py * W + px]) : 0.f;
    }
    __syncthreads();

    // ---- window gradients of the warp's group
    float4 gk[4];
    CbGroup g;
    int ux = 0x7fffffff, uy = 0x7fffffff, vx = -0x7fffffff, vy = -0x7fffffff;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      gk[k] = geo[(gy + (k >> 1)) * 8 + gx + (k & 1)];
      const int xw = __float_as_int(gk[k].z), yw = __float_as_int(gk[k].w);
      const int xa = max(xw, 0), ya = max(yw, 0), xe = min(xw + D, W2), ye = min(yw + D, H2);
      if (xa < xe && ya < ye) {
        ux = min(ux, xa);
        uy = min(uy, ya);
        vx = max(vx, xe);
        vy = max(vy, ye);
      }
    }
    g.x0 = ux;
    g.y0 = uy;
    g.w = ux < vx ? vx - ux : 0;
    g.h = uy < vy ? vy - uy : 0;
    const int npos = g.w * g.h;
    g.mode = npos == 0 ? 0 : (!separate && npos <= A.cap) ? 1 : 2;
    if (lane == 0) grp[warp] = g;
    // the blend's adjoint at tap (px, py) of pixel k, 0 outside its window
    auto adjoint = [&](int k, int px, int py) -> float {
      if (px < 0 || px >= D || py < 0 || py >= D) return 0.f;
      const float dx = gk[k].x, dy = gk[k].y;
      const float* row = gs + ((gy + (k >> 1)) * 8 + gx + (k & 1)) * gst;
      float s = 0.f;
      if (px < rd && py < rd) s += (1.f - dx) * (1.f - dy) * row[px * rd + py];
      if (px > 0 && py < rd) s += dx * (1.f - dy) * row[(px - 1) * rd + py];
      if (px < rd && py > 0) s += (1.f - dx) * dy * row[px * rd + py - 1];
      if (px > 0 && py > 0) s += dx * dy * row[(px - 1) * rd + py - 1];
      return s;
    };
    float4* gw = Gu + warp * A.cap;
    float* gw1 = reinterpret_cast<float*>(gw);                     // mode 2: [4][D][D]
    if (g.mode == 1) {
      for (int p = lane; p < npos; p += 32) {
        const int yy = p / g.w, x = ux + p - yy * g.w, y = uy + yy;
        float4 v;
        v.x = adjoint(0, x - __float_as_int(gk[0].z), y - __float_as_int(gk[0].w));
        v.y = adjoint(1, x - __float_as_int(gk[1].z), y - __float_as_int(gk[1].w));
        v.z = adjoint(2, x - __float_as_int(gk[2].z), y - __float_as_int(gk[2].w));
        v.w = adjoint(3, x - __float_as_int(gk[3].z), y - __float_as_int(gk[3].w));
        gw[p] = v;
      }
    } else if (g.mode == 2) {
      for (int t = lane; t < D * D; t += 32) {
        const int py = t / D, px = t - py * D;
#pragma unroll
        for (int k = 0; k < 4; ++k) gw1[k * D * D + t] = adjoint(k, px, py);
      }
    }
    __syncthreads();

    // ---- the tile's f1 rows, for g2 (over the staged gradients)
    for (int idx = tid; idx < 64 * 32; idx += kCbThreads) {
      const int q = idx >> 5, px = tx0 + (q & 7), py = ty0 + (q >> 3);
      F1[idx] = (px < W && py < H) ? __ldg(f1 + (int64_t)(py * W + px) * 32 + (idx & 31)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    // ---- g1: one warp per group
    {
      float4 acc[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[k] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (g.mode == 1) {
        for (int yy = 0; yy < g.h; ++yy) {
          const float4* row = f2 + ((int64_t)(uy + yy) * W2 + ux) * 32 + lane;
          const float4* gp = gw + yy * g.w;
#pragma unroll 4
          for (int x = 0; x < g.w; ++x) {
            const float4 v = __ldg(row + x * 32), c = gp[x];
            fma4(acc[0], c.x, v);
            fma4(acc[1], c.y, v);
            fma4(acc[2], c.z, v);
            fma4(acc[3], c.w, v);
          }
        }
      } else if (g.mode == 2) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int xw = __float_as_int(gk[k].z), yw = __float_as_int(gk[k].w);
          const int xa = max(xw, 0), xe = min(xw + D, W2), ye = min(yw + D, H2);
          for (int y = max(yw, 0); y < ye; ++y)
            for (int x = xa; x < xe; ++x)
              fma4(acc[k], gw1[k * D * D + (y - yw) * D + x - xw], __ldg(f2 + ((int64_t)y * W2 + x) * 32 + lane));
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int px = tx0 + gx + (k & 1), py = ty0 + gy + (k >> 1);
        if (px >= W || py >= H) continue;
        float4* dst = o1 + (int64_t)(py * W + px) * 32 + lane;
        if (kRed1) {
          red4(reinterpret_cast<float*>(dst), acc[k]);
        } else if (lvl == 0) {
          *dst = acc[k];
        } else {
          const float4 old = *dst;
          *dst = make_float4(old.x + acc[k].x, old.y + acc[k].y, old.z + acc[k].z, old.w + acc[k].w);
        }
      }
    }
    __syncthreads();

    // ---- g2: one warp per 2x2 block of the tile's box
    CbGroup mine{0, 0, 0, 0, 0};
    if (lane < 16) mine = grp[lane];
    int bx0 = mine.mode ? mine.x0 : 0x7fffffff, by0 = mine.mode ? mine.y0 : 0x7fffffff;
    int bx1 = mine.mode ? mine.x0 + mine.w : -1, by1 = mine.mode ? mine.y0 + mine.h : -1;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      bx0 = min(bx0, __shfl_xor_sync(0xffffffffu, bx0, o));
      by0 = min(by0, __shfl_xor_sync(0xffffffffu, by0, o));
      bx1 = max(bx1, __shfl_xor_sync(0xffffffffu, bx1, o));
      by1 = max(by1, __shfl_xor_sync(0xffffffffu, by1, o));
    }
    bx0 = __shfl_sync(0xffffffffu, bx0, 0);
    by0 = __shfl_sync(0xffffffffu, by0, 0);
    bx1 = __shfl_sync(0xffffffffu, bx1, 0);
    by1 = __shfl_sync(0xffffffffu, by1, 0);
    const int nbx = bx1 > bx0 ? (bx1 - bx0 + 1) / 2 : 0, nby = by1 > by0 ? (by1 - by0 + 1) / 2 : 0;
    for (int blk = warp; blk < nbx * nby; blk += kCbThreads / 32) {
      const int qy = blk / nbx, x = bx0 + 2 * (blk - qy * nbx), y = by0 + 2 * qy;
      const bool hit = mine.mode && x + 1 >= mine.x0 && x < mine.x0 + mine.w && y + 1 >= mine.y0 && y < mine.y0 + mine.h;
      unsigned mask = __ballot_sync(0xffffffffu, hit);
      if (!mask) continue;
      float4 acc[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[j] = make_float4(0.f, 0.f, 0.f, 0.f);
      for (; mask; mask &= mask - 1) {
        const int gi = __ffs(mask) - 1;
        const CbGroup q = grp[gi];
        const float4* fq = F1 + ((2 * (gi >> 2)) * 8 + 2 * (gi & 3)) * 32 + lane;
        if (q.mode == 1) {
          const float4* gp = Gu + gi * A.cap + (y - q.y0) * q.w + x - q.x0;
          const bool xa = x >= q.x0, xb = x + 1 < q.x0 + q.w, ya = y >= q.y0, yb = y + 1 < q.y0 + q.h;
          const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
          float4 c[4];
          c[0] = xa && ya ? gp[0] : zero;
          c[1] = xb && ya ? gp[1] : zero;
          c[2] = xa && yb ? gp[q.w] : zero;
          c[3] = xb && yb ? gp[q.w + 1] : zero;
          float4 v = fq[0];
#pragma unroll
          for (int j = 0; j < 4; ++j) fma4(acc[j], c[j].x, v);
          v = fq[32];
#pragma unroll
          for (int j = 0; j < 4; ++j) fma4(acc[j], c[j].y, v);
          v = fq[8 * 32];
#pragma unroll
          for (int j = 0; j < 4; ++j) fma4(acc[j], c[j].z, v);
          v = fq[9 * 32];
#pragma unroll
          for (int j = 0; j < 4; ++j) fma4(acc[j], c[j].w, v);
        } else {
          const float* gp = reinterpret_cast<const float*>(Gu + gi * A.cap);
          for (int k = 0; k < 4; ++k) {
            const float4 e = geo[((gi >> 2) * 2 + (k >> 1)) * 8 + 2 * (gi & 3) + (k & 1)];
            const int wx = x - __float_as_int(e.z), wy = y - __float_as_int(e.w);
            const float4 v = fq[((k >> 1) * 8 + (k & 1)) * 32];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const int tx = wx + (j & 1), ty = wy + (j >> 1);
              if (tx < 0 || tx >= D || ty < 0 || ty >= D) continue;
              const float c = gp[k * D * D + ty * D + tx];
              if (c != 0.f) fma4(acc[j], c, v);   // a zero gradient adds nothing, whatever the feature
            }
          }
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int xx = x + (j & 1), yy = y + (j >> 1);
        if (xx < W2 && yy < H2) red4(o2 + ((int64_t)yy * W2 + xx) * kCbC + 4 * lane, acc[j]);
      }
    }
  }
}

// Where the frames that the edges use are packed: slot[f] = their number below f, -1 for a frame that
// no edge uses; CTA 0 for the edges' ii, CTA 1 for jj.  At most m slots a side.
__global__ void __launch_bounds__(1024)
corr_bwd_slots_kernel(const int64_t* __restrict__ ii, const int64_t* __restrict__ jj, int m, int n1, int n2,
                      int* __restrict__ slot1, int* __restrict__ slot2) {
  const int64_t* idx = blockIdx.x ? jj : ii;
  const int n = blockIdx.x ? n2 : n1, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int* slot = blockIdx.x ? slot2 : slot1;
  __shared__ int counts[32];
  for (int f = tid; f < n; f += 1024) slot[f] = 0;
  __syncthreads();
  for (int e = tid; e < m; e += 1024) {
    const int64_t f = idx[e];
    if (f >= 0 && f < n) slot[f] = 1;
  }
  __syncthreads();
  int base = 0;
  for (int f0 = 0; f0 < n; f0 += 1024) {
    const int f = f0 + tid;
    const bool used = f < n && slot[f];
    const unsigned mask = __ballot_sync(0xffffffffu, used);
    if (lane == 0) counts[warp] = __popc(mask);
    __syncthreads();
    int at = base;
    for (int q = 0; q < 32; ++q) {
      if (q < warp) at += counts[q];
      base += counts[q];
    }
    if (f < n) slot[f] = used ? at + __popc(mask & ((1u << lane) - 1)) : -1;
    __syncthreads();
  }
}

// channel-first features of the frames in use -> FP32 channel-last, their accumulators
// zeroed; sets *nonfinite when a feature is not finite
template <typename T>
__global__ void __launch_bounds__(256)
corr_bwd_pack_kernel(const T* __restrict__ src, float* __restrict__ dst, float* __restrict__ acc,
                     const int* __restrict__ slots, int N, int S, int HW, int32_t* __restrict__ nonfinite) {
  __shared__ float tile[kCbPackPix][kCbC + 1];
  const int n = blockIdx.y, slot = slots ? slots[n] : n;
  if (slot < 0) return;
  const int p0 = blockIdx.x * kCbPackPix, np = min(kCbPackPix, HW - p0);
  const int64_t frame = (int64_t)blockIdx.z * S + slot;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const T* s = src + ((int64_t)blockIdx.z * N + n) * kCbC * HW + p0;
  const int q = threadIdx.x & (kCbPackPix - 1), cq = threadIdx.x / kCbPackPix;
  bool bad = false;
  if (q < np) {
#pragma unroll 2
    for (int c0 = cq; c0 < kCbC; c0 += 8 * kCbPackCh) {       // eight loads in flight, twice
      T v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = s[(int64_t)(c0 + i * kCbPackCh) * HW + q];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float f = to_f(v[i]);
        bad |= !isfinite(f);
        tile[q][c0 + i * kCbPackCh] = f;
      }
    }
  }
  if (bad) atomicOr(nonfinite, 1);
  __syncthreads();
  float* d = dst + (frame * HW + p0) * kCbC + lane;
#pragma unroll 4
  for (int p = warp; p < np; p += 8) {                        // a pixel's row by one warp
#pragma unroll
    for (int k = 0; k < kCbC; k += 32) d[p * kCbC + k] = tile[p][lane + k];
  }
  if (acc) {
    float4* a = reinterpret_cast<float4*>(acc + (frame * HW + p0) * kCbC);
    for (int i = threadIdx.x; i < np * (kCbC / 4); i += 256) a[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

// 2x2 average of a channel-last level (rows of 128 floats), as avg_pool2d sums it; the level's
// gradient accumulator is zeroed.  One warp per output position.
__global__ void __launch_bounds__(256)
corr_bwd_pool_kernel(const float* __restrict__ src, float* __restrict__ dst, float* __restrict__ acc, int H, int W,
                     int64_t total) {
  const int H2 = H >> 1, W2 = W >> 1, lane = threadIdx.x & 31;
  const int64_t at = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (at >= total) return;
  const int64_t n = at / (H2 * W2);
  const int rem = (int)(at - n * (H2 * W2)), y = rem / W2, x = rem - y * W2;
  const float4* s = reinterpret_cast<const float4*>(src) + ((n * H + 2 * y) * W + 2 * x) * 32 + lane;
  const float4 a = s[0], b = s[32], c = s[(int64_t)W * 32], d = s[(int64_t)W * 32 + 32];
  reinterpret_cast<float4*>(dst)[at * 32 + lane] =
      make_float4((a.x + b.x + c.x + d.x) * 0.25f, (a.y + b.y + c.y + d.y) * 0.25f, (a.z + b.z + c.z + d.z) * 0.25f,
                  (a.w + b.w + c.w + d.w) * 0.25f);
  reinterpret_cast<float4*>(acc)[at * 32 + lane] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// FP32 channel-last accumulators -> channel-first gradients of T; frames out of use give 0.
// With levels > 1 the gradients of the 2x2-averaged levels come back to their pixels (a
// quarter of the level above's, which holds a quarter of the next).
struct CbUnpack {
  const float* acc[4];
  int levels, H[4], W[4];
};
template <typename T>
__global__ void __launch_bounds__(256)
corr_bwd_unpack_kernel(const __grid_constant__ CbUnpack U, T* __restrict__ dst,
                       const int* __restrict__ slots, int N, int S) {
  __shared__ float tile[kCbPackPix][kCbC + 1];
  const int n = blockIdx.y, slot = slots ? slots[n] : n, W = U.W[0], HW = U.H[0] * W;
  const int p0 = blockIdx.x * kCbPackPix, np = min(kCbPackPix, HW - p0);
  const int64_t frame = (int64_t)blockIdx.z * S + slot;
  if (slot < 0) {
    // no edge uses the frame: its share of the frame's zeros, by 16-byte stores where they are aligned
    T* f = dst + ((int64_t)blockIdx.z * N + n) * kCbC * HW + (int64_t)blockIdx.x * kCbPackPix * kCbC;
    const int count = np * kCbC;              // of 128 HW elements: the blocks' runs are equal but for the last
    constexpr int kVec = 16 / sizeof(T);
    if (reinterpret_cast<uintptr_t>(f) & 15) {
      for (int i = threadIdx.x; i < count; i += 256) f[i] = from_f<T>(0.f);
    } else {
      for (int i = threadIdx.x; i < count / kVec; i += 256) reinterpret_cast<uint4*>(f)[i] = make_uint4(0, 0, 0, 0);
    }
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll 2
  for (int q = warp; q < np; q += 8) {                        // a pixel's row by one warp, all levels' loads together
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    const int y = (p0 + q) / W, x = (p0 + q) - y * W;
    float a[4][4];
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      if (l < U.levels) {
        const int yl = y >> l, xl = x >> l;
        const bool in = yl < U.H[l] && xl < U.W[l];
        const float* row = U.acc[l] + ((frame * U.H[l] + yl) * U.W[l] + xl) * kCbC + lane;
#pragma unroll
        for (int k = 0; k < 4; ++k) a[l][k] = in ? row[32 * k] : 0.f;
      }
    }
#pragma unroll
    for (int l = 3; l >= 0; --l) {
      if (l < U.levels) {
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = (v[k] + a[l][k]) * (l > 0 ? 0.25f : 1.f);
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) tile[q][lane + 32 * k] = v[k];
  }
  __syncthreads();
  T* d = dst + ((int64_t)blockIdx.z * N + n) * kCbC * HW + p0;
  const int q = threadIdx.x & (kCbPackPix - 1), cq = threadIdx.x / kCbPackPix;
  if (q < np) {
#pragma unroll 8
    for (int c = cq; c < kCbC; c += kCbPackCh) d[(int64_t)c * HW + q] = from_f<T>(tile[q][c]);
  }
}

template <typename TG, bool kRed1>
int cb_tile(const CbArgs& a, int b, cudaStream_t s) {
  static DeviceOnce once;
  int dev = 0;
  HS2_CUDA(cudaGetDevice(&dev));
  int rc = once.run(dev, [&]() -> int {
    HS2_CUDA(cudaFuncSetAttribute(corr_bwd_tile_kernel<TG, kRed1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)cb_smem(kCbMaxRadius)));
    return HS2_OK;
  });
  if (rc) return rc;
  dim3 grid(((a.W + 7) / 8) * ((a.H + 7) / 8), a.M, b);
  HS2_PROF("corr_bwd_tile", s);
  corr_bwd_tile_kernel<TG, kRed1><<<grid, kCbThreads, cb_smem(a.r), s>>>(a);
  HS2_LAUNCH_CHECK("corr_bwd_tile_kernel");
  return HS2_OK;
}

size_t up256(size_t n) { return (n + 255) & ~(size_t)255; }

template <typename T>
int cb_pack(const void* src, float* dst, float* acc, const int* slots, int b, int n, int cap, int hw, int32_t* bad,
            cudaStream_t s) {
  HS2_PROF("corr_bwd_pack", s);
  corr_bwd_pack_kernel<T><<<dim3((hw + kCbPackPix - 1) / kCbPackPix, n, b), 256, 0, s>>>(static_cast<const T*>(src), dst,
                                                                                       acc, slots, n, cap, hw, bad);
  HS2_LAUNCH_CHECK("corr_bwd_pack_kernel");
  return HS2_OK;
}

template <typename T>
int cb_unpack(const CbUnpack& u, void* dst, const int* slots, int b, int n, int cap, cudaStream_t s) {
  HS2_PROF("corr_bwd_unpack", s);
  corr_bwd_unpack_kernel<T><<<dim3((u.H[0] * u.W[0] + kCbPackPix - 1) / kCbPackPix, n, b), 256, 0, s>>>(
      u, static_cast<T*>(dst), slots, n, cap);
  HS2_LAUNCH_CHECK("corr_bwd_unpack_kernel");
  return HS2_OK;
}

template <typename T>
int altcorr_bwd_tiled_t(const void* fmap1, const void* fmap2, int b, int n1, int n2, int h, int w, int h2, int w2,
                        const float* coords, const int64_t* ii, const int64_t* jj, int m, const float* grad,
                        int radius, float scale, void* g1, void* g2, int32_t* info, void* ws, cudaStream_t s) {
  const int s1 = std::min(n1, m), s2 = std::min(n2, m);
  const size_t e1 = up256((size_t)b * s1 * h * w * kCbC * 4), e2 = up256((size_t)b * s2 * h2 * w2 * kCbC * 4);
  char* p = static_cast<char*>(ws);
  float *f1 = reinterpret_cast<float*>(p), *f2 = reinterpret_cast<float*>(p + e1);
  float *o1 = reinterpret_cast<float*>(p + e1 + e2), *o2 = reinterpret_cast<float*>(p + 2 * e1 + e2);
  int32_t* bad = reinterpret_cast<int32_t*>(p + 2 * (e1 + e2));
  int *slot1 = bad + 1, *slot2 = slot1 + n1;
  HS2_CUDA(cudaMemsetAsync(bad, 0, sizeof(int32_t), s));
  corr_bwd_slots_kernel<<<2, 1024, 0, s>>>(ii, jj, m, n1, n2, slot1, slot2);
  HS2_LAUNCH_CHECK("corr_bwd_slots_kernel");
  int rc;
  if ((rc = cb_pack<T>(fmap1, f1, o1, slot1, b, n1, s1, h * w, bad, s))) return rc;
  if ((rc = cb_pack<T>(fmap2, f2, o2, slot2, b, n2, s2, h2 * w2, bad, s))) return rc;
  CbArgs a{};
  a.f1 = f1;
  a.f2[0] = f2;
  a.o1 = o1;
  a.o2[0] = o2;
  a.coords = coords;
  a.grad = grad;
  a.ii = ii;
  a.jj = jj;
  a.slot1 = slot1, a.slot2 = slot2, a.S1 = s1, a.S2 = s2;
  a.N1 = n1, a.N2 = n2, a.M = m, a.H = h, a.W = w, a.r = radius, a.levels = 1, a.cap = cb_cap(radius);
  a.H2[0] = h2, a.W2[0] = w2;
  a.scale = scale;
  a.nonfinite = bad;
  a.info = info;
  if ((rc = cb_tile<float, true>(a, b, s))) return rc;
  CbUnpack u{};
  u.levels = 1;
  u.acc[0] = o1, u.H[0] = h, u.W[0] = w;
  if ((rc = cb_unpack<T>(u, g1, slot1, b, n1, s1, s))) return rc;
  u.acc[0] = o2, u.H[0] = h2, u.W[0] = w2;
  return cb_unpack<T>(u, g2, slot2, b, n2, s2, s);
}

// Workspace of the lookup's backward: packed fmap1 and its accumulator, then per level the packed
// (pooled) fmap2 and its accumulator, then the non-finite flag.
struct ClLayout {
  size_t f1, o1, f2[4], o2[4], flag, total;
};
ClLayout cl_layout(int64_t n, int h, int w, int levels) {
  ClLayout L{};
  size_t o = 0;
  auto take = [&](size_t bytes) { const size_t at = o; o += up256(bytes); return at; };
  const size_t row = kCbC * 4;
  L.f1 = take(n * h * w * row);
  L.o1 = take(n * h * w * row);
  for (int l = 0; l < levels; ++l) {
    L.f2[l] = take(n * (h >> l) * (w >> l) * row);
    L.o2[l] = take(n * (h >> l) * (w >> l) * row);
  }
  L.flag = take(256);
  L.total = o;
  return L;
}

template <typename T>
int corr_lookup_bwd_t(const void* fmap1, const void* fmap2, int n, int h, int w, const float* coords, const void* grad,
                      int levels, int radius, float scale, void* g1, void* g2, char* ws, cudaStream_t s) {
  const ClLayout L = cl_layout(n, h, w, levels);
  auto at = [&](size_t o) { return reinterpret_cast<float*>(ws + o); };
  int32_t* bad = reinterpret_cast<int32_t*>(ws + L.flag);
  HS2_CUDA(cudaMemsetAsync(bad, 0, sizeof(int32_t), s));
  int rc;
  if ((rc = cb_pack<T>(fmap1, at(L.f1), nullptr, nullptr, 1, n, n, h * w, bad, s))) return rc;
  if ((rc = cb_pack<T>(fmap2, at(L.f2[0]), at(L.o2[0]), nullptr, 1, n, n, h * w, bad, s))) return rc;
  for (int l = 1; l < levels; ++l) {
    const int64_t total = (int64_t)n * (h >> l) * (w >> l);
    HS2_PROF("corr_bwd_pool", s);
    corr_bwd_pool_kernel<<<(unsigned)((total + 7) / 8), 256, 0, s>>>(at(L.f2[l - 1]), at(L.f2[l]), at(L.o2[l]),
                                                                   h >> (l - 1), w >> (l - 1), total);
    HS2_LAUNCH_CHECK("corr_bwd_pool_kernel");
  }
  CbArgs a{};
  a.f1 = at(L.f1);
  a.o1 = at(L.o1);
  a.coords = coords;
  a.interleaved = 1;
  a.grad = grad;
  a.N1 = a.N2 = a.S1 = a.S2 = a.M = n, a.H = h, a.W = w, a.r = radius, a.levels = levels, a.cap = cb_cap(radius);
  a.scale = scale;
  a.nonfinite = bad;
  CbUnpack u{};
  u.levels = levels;
  for (int l = 0; l < levels; ++l) {
    a.f2[l] = at(L.f2[l]);
    a.o2[l] = at(L.o2[l]);
    a.H2[l] = u.H[l] = h >> l;
    a.W2[l] = u.W[l] = w >> l;
    u.acc[l] = at(L.o2[l]);
  }
  if ((rc = cb_tile<T, false>(a, 1, s))) return rc;
  if ((rc = cb_unpack<T>(u, g2, nullptr, 1, n, n, s))) return rc;
  u.levels = 1;
  u.acc[0] = at(L.o1);
  return cb_unpack<T>(u, g1, nullptr, 1, n, n, s);
}

int cl_check(int dtype, int n, int c, int h, int w, int levels, int radius) {
  if (dtype != HS2_F32 && dtype != HS2_F16 && dtype != HS2_BF16) {
    set_error("corr_lookup_backward: unsupported dtype %d (f32, f16, bf16)", dtype);
    return HS2_ERR_DTYPE;
  }
  if (n < 0 || n > 65535 || c != kCbC || h <= 0 || w <= 0 || levels < 1 || levels > 4 || (h >> (levels - 1)) < 1 ||
      (w >> (levels - 1)) < 1 || radius < 0 || radius > kCbMaxRadius || (int64_t)h * w > (1 << 24)) {
    set_error("corr_lookup_backward: bad sizes n=%d c=%d h=%d w=%d levels=%d r=%d (128 channels, 1 to 4 levels, "
              "radius <= %d)", n, c, h, w, levels, radius, kCbMaxRadius);
    return HS2_ERR_INVALID;
  }
  return HS2_OK;
}

}  // namespace

bool altcorr_bwd_tiled_ok(int b, int n1, int n2, int c, int m, int radius) {
  return c == kCbC && radius <= kCbMaxRadius && b > 0 && n1 > 0 && n2 > 0 && n1 <= 65535 && n2 <= 65535 && m > 0;
}

size_t altcorr_bwd_tiled_bytes(int b, int n1, int n2, int h, int w, int h2, int w2, int m) {
  return 2 * (up256((size_t)b * std::min(n1, m) * h * w * kCbC * 4) +
              up256((size_t)b * std::min(n2, m) * h2 * w2 * kCbC * 4)) +
         up256(((size_t)n1 + n2 + 1) * sizeof(int32_t));
}

int altcorr_bwd_tiled(int dtype, const void* fmap1, const void* fmap2, int b, int n1, int n2, int h, int w, int h2,
                      int w2, const float* coords, const int64_t* ii, const int64_t* jj, int m, const float* grad,
                      int radius, float scale, void* g1, void* g2, int32_t* info, void* ws, cudaStream_t s) {
  switch (dtype) {
    case HS2_F32:
      return altcorr_bwd_tiled_t<float>(fmap1, fmap2, b, n1, n2, h, w, h2, w2, coords, ii, jj, m, grad, radius, scale,
                                        g1, g2, info, ws, s);
    case HS2_F16:
      return altcorr_bwd_tiled_t<__half>(fmap1, fmap2, b, n1, n2, h, w, h2, w2, coords, ii, jj, m, grad, radius, scale,
                                         g1, g2, info, ws, s);
    default:
      return altcorr_bwd_tiled_t<__nv_bfloat16>(fmap1, fmap2, b, n1, n2, h, w, h2, w2, coords, ii, jj, m, grad, radius,
                                                scale, g1, g2, info, ws, s);
  }
}

}  // namespace hs2

extern "C" int hs2_corr_lookup_backward_workspace_size(int dtype, int n, int c, int h, int w, int levels, int radius,
                                                       size_t* bytes) {
  using namespace hs2;
  if (!bytes) {
    set_error("corr_lookup_backward_workspace_size: null output");
    return HS2_ERR_INVALID;
  }
  const int rc = cl_check(dtype, n, c, h, w, levels, radius);
  if (rc) return rc;
  *bytes = cl_layout(n, h, w, levels).total;
  return HS2_OK;
}

extern "C" int hs2_corr_lookup_backward(const void* fmap1, const void* fmap2, int dtype, int n, int c, int h, int w,
                                        const float* coords, const void* grad, int levels, int radius, float scale,
                                        void* fmap1_grad, void* fmap2_grad, void* workspace, size_t workspace_bytes,
                                        hs2_stream_t stream) {
  using namespace hs2;
  int rc = cl_check(dtype, n, c, h, w, levels, radius);
  if (rc) return rc;
  if (n == 0) return HS2_OK;
  if (!fmap1 || !fmap2 || !coords || !grad || !fmap1_grad || !fmap2_grad) {
    set_error("corr_lookup_backward: null pointer argument");
    return HS2_ERR_INVALID;
  }
  const size_t need = cl_layout(n, h, w, levels).total;
  if (!workspace || workspace_bytes < need) {
    set_error("corr_lookup_backward: workspace of %zu bytes required", need);
    return HS2_ERR_WORKSPACE;
  }
  if (reinterpret_cast<uintptr_t>(workspace) & 15) {
    set_error("corr_lookup_backward: the workspace must start on a 16-byte boundary");
    return HS2_ERR_WORKSPACE;
  }
  if ((rc = bind_device(fmap1_grad))) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  char* ws = static_cast<char*>(workspace);
  if (dtype == HS2_F32)
    return corr_lookup_bwd_t<float>(fmap1, fmap2, n, h, w, coords, grad, levels, radius, scale, fmap1_grad, fmap2_grad, ws, s);
  if (dtype == HS2_F16)
    return corr_lookup_bwd_t<__half>(fmap1, fmap2, n, h, w, coords, grad, levels, radius, scale, fmap1_grad, fmap2_grad, ws, s);
  return corr_lookup_bwd_t<__nv_bfloat16>(fmap1, fmap2, n, h, w, coords, grad, levels, radius, scale, fmap1_grad, fmap2_grad,
                                          ws, s);
}
