// Mono-prior depth / scale alignment step: HI-SLAM2's JDSA (hislam2/geom/ba.py:170-219 with
// get_prior_depth_aligned :159-167 and geom/chol.py:schur_solve_mono_prior :80-107).
//
// The reference builds the step from dense tensors: the bilinear scale Jacobian [M,H,W,hs,ws],
// E [M*D, M*HW] (D = hs*ws scale unknowns per frame), E Q E^T and one Cholesky of the
// [M*D, M*D] system, then inv(L) E Q for the depth covariance.  Its scatter keys are
// (kx', kx') with kx' = kx - kx[0] (kx = unique(ii)), so H and E only have diagonal blocks:
// the reduced system is block diagonal, one D x D block per source frame, and the whole
// step is per frame.  Block b couples the prior terms of frame kx[0] + b (when that frame
// is a source frame; else none) with row b of C, w, eta and the prior mask (frame kx[b]):
// the two are the same frame whenever kx is contiguous, and this pairing is what the
// reference computes when it is not.
//
//   jdsa_keys          kx and slot of the edges from a bitmap of the frames, one CTA: a list of a
//                      few hundred edges needs no sort, and the count stays on the device;
//   proj_trans         (geometry.cu) windows of more than kJdFusedBlocks source frames: the depth-only
//                      Schur terms C, w, edge by edge with atomics, ahead of a jdsa_step that reads them;
//   jdsa_step          cluster of 8 (after proj_trans: 2) CTAs per block b, pixels dealt out in runs of
//                      a CTA: per pixel the depth-only Schur terms C, w summed over the block's
//                      edges in their order (proj_trans's terms); then, in FP32 as the reference,
//                        Q = 1 / (C + m alpha + (1 - m) eta),  w' = w - m alpha rd,
//                        a = prior [> 0] of the source frame, J = -a (wa, wb, wc, wd) at the
//                        pixel's interpolation cell,
//                      summed in FP64 per cell over the cluster: S += alpha a^2 (1 - alpha Q) w w^T,
//                      diag(H) += alpha a^2 w^2, v += alpha a w (rd_src + Q w'); then
//                      S + diag(0.1 + 1e-4 diag(H)) = L L^T in FP64 by one warp (D <= 16),
//                      dso = S^-1 v; second pass: dz = Q (w' + alpha a (w . dso_cell)),
//                      disps_out = clamp(where(d + dz > 10, 0, d + dz), min = 0.001) and
//                      dzcov = (alpha a Q)^2 w^T S^-1_cell w + Q  (= |L^-1 E Q|^2 + Q).
//                      The clusters behind the M blocks copy the frames that are not source
//                      frames through the same where / clamp (the reference applies both to
//                      the whole window).
//   jdsa_scales        dscales[kx[b]] += dso[b], skipped when a block was not positive
//                      definite or an index was bad (the reference raises before it).
//
// Bound by latency: 25 frames of 3311 pixels are 14 MB, 2 us of HBM.  One CTA per frame took
// 13 pixels a thread through two passes behind a launch of atomics that summed C and w; eight
// CTAs a frame take two pixels a thread, keep the sums of an edge list they scan themselves
// (no zeroed buffers, no atomics, a fixed order) and meet once, in distributed shared memory.
// 25 frames at 43x77, 258 edges, 2x2 grid: a call of mono.JDSA 183 -> 121 us (most of it the
// keys, which torch.unique made behind two waits of the host; the kernels 61 -> 53 us), of
// which the host's own work is half.
#include <utility>

#include <cooperative_groups.h>

#include "common.cuh"
#include "profile.cuh"

namespace hs2 {

namespace {

constexpr int kJdThreads = 256;
constexpr int kJdWarps = kJdThreads / 32;
// Up to kJdFusedBlocks source frames (two waves of their CTAs) a cluster of eight CTAs sums its block's
// edges itself.  Each of its CTAs looks through the whole edge list, so beyond that proj_trans
// sums them, a CTA per edge, and two CTAs a block have work enough for the GPU.  A call, the edges summed
// by the cluster / ahead: 60 frames of 43x77 with 700 edges 140 / 146 us, 100 with 2000 234 / 181, 300
// with 6000 546 / 333, 1000 of 24x32 with 20000 2030 / 335; 150 of 120x160 with 2000 575 / 504.
constexpr int kJdCluster = 8;      // the portable cluster size
constexpr int kJdPlainCluster = 2;
constexpr int kJdFusedBlocks = 2 * 2 * kNumSMs / kJdCluster;
constexpr int kJdBatch = 64;       // edges whose relative poses are in shared memory at a time
constexpr int kJdMaxD = 16;
constexpr int kJdMaxCells = 9;     // (hs - 1)(ws - 1) for hs ws <= 16
constexpr int kJdSums = 18;        // one cell: 10 Gram terms, 4 diag(H) terms, 4 rhs terms
constexpr int kJdMaxAxis = 4096;   // ht, wd (the grid axes are staged in shared memory)
constexpr double kJdEp = 0.1;      // schur_solve_mono_prior's ep and lm (chol.py:80)
constexpr double kJdLm = 1e-4;
constexpr int kJdKeyThreads = 1024;
constexpr int kJdKeyFrames = 65536;   // frames of the bitmap (8 KB of shared memory)
constexpr unsigned kJdCopyClusters = 1024;

struct JdArgs {
  const float* poses;
  int64_t num_poses;
  const float* intr;
  const float* targets;
  const float* weights;
  const int64_t* ii;
  const int64_t* jj;
  const int64_t* slot;
  int64_t num_edges;
  const float* disps;
  int64_t num_disps;
  int ht, wd;
  float* C;   // a pixel's sums are written and read by one thread
  float* w;
  const float* eta;
  const float* prior;
  int64_t num_prior;
  const float* dscales;
  int64_t num_scales;
  int hs, ws;
  const float* gy;
  const float* gx;
  const int64_t* kx;
  int M;
  float alpha;
  float* dso;     // [M, D]
  float* out;     // [num_disps, H, W]
  float* dzcov;   // [M, HW] or null
  int32_t* info;
};

__device__ __forceinline__ int find_sorted(const int64_t* kx, int M, int64_t f) {
  int lo = 0, hi = M - 1;
  while (lo <= hi) {
    const int mid = (lo + hi) >> 1;
    const int64_t v = kx[mid];
    if (v == f) return mid;
    if (v < f) lo = mid + 1;
    else hi = mid - 1;
  }
  return -1;
}

// torch.where(d > 10, 0, d).clamp(min=0.001); NaN passes through as in torch
__device__ __forceinline__ float jd_clean(float d) {
  d = d > 10.f ? 0.f : d;
  return d < 0.001f ? 0.001f : d;
}

// One pixel's interpolation cell: bi_inter_kernel's weights (droid_kernels.cu:1297-1306)
// and the D-indices of the corners (y0,x0), (y1,x0), (y0,x1), (y1,x1) they multiply.
struct Cell {
  float wt[4];
  int pos[4];
};

__device__ __forceinline__ Cell make_cell(float x, float y, int cx, int cy, int ws) {
  const float x0 = (float)cx, y0 = (float)cy, x1 = x0 + 1.f, y1 = y0 + 1.f;
  Cell c;
  c.wt[0] = (x1 - x) * (y1 - y);
  c.wt[1] = (x1 - x) * (y - y0);
  c.wt[2] = (x - x0) * (y1 - y);
  c.wt[3] = (x - x0) * (y - y0);
  c.pos[0] = cy * ws + cx;
  c.pos[1] = (cy + 1) * ws + cx;
  c.pos[2] = cy * ws + cx + 1;
  c.pos[3] = (cy + 1) * ws + cx + 1;
  return c;
}

__device__ __forceinline__ float interp(const float* S, const Cell& c) {
  return c.wt[0] * S[c.pos[0]] + c.wt[1] * S[c.pos[1]] + c.wt[2] * S[c.pos[2]] + c.wt[3] * S[c.pos[3]];
}

// Row terms of pixel k of block b (frame fr): Q, w' and the disparity itself.
struct RowTerms {
  float Q, wq, d;
};

__device__ __forceinline__ RowTerms row_terms(const JdArgs& A, int b, int64_t fr, int HW, int k, const float* sc,
                                              const Cell& c) {
  const int64_t rk = (int64_t)b * HW + k, fk = fr * HW + k;
  const float pr = A.prior[fk];
  const float m = pr > 0.f ? 1.f : 0.f;
  const float d = A.disps[fk];
  const float rd = d - pr * interp(sc, c);
  const float Cb = A.C[rk] + m * A.alpha + (1.f - m) * A.eta[rk];
  RowTerms t;
  t.Q = 1.0f / Cb;
  t.wq = A.w[rk] - m * A.alpha * rd;
  t.d = d;
  return t;
}

// An edge of the block as its pixels need it: Gij as a matrix and the disparities of its source frame.
struct JdEdge {
  float t[3], R[9];
  int e;
  const float* d;
};

// An edge outside the buffers marks the step as invalid and stands for frame fr, identity: nothing
// is read out of bounds and the loop over the edges needs no test.
__device__ __forceinline__ JdEdge load_edge(const JdArgs& A, int e, int64_t fr, int HW) {
  JdEdge g;
  const int64_t ix = A.ii[e], jx = A.jj[e];
  if (ix < 0 || jx < 0 || ix >= A.num_poses || jx >= A.num_poses || ix >= A.num_disps) {
    atomicOr(A.info, HS2_DEV_BAD_INDEX);
    for (int i = 0; i < 3; ++i) g.t[i] = 0.f;
    for (int i = 0; i < 9; ++i) g.R[i] = i % 4 ? 0.f : 1.f;
    g.e = e;
    g.d = A.disps + fr * HW;
    return g;
  }
  const float* pi = A.poses + 7 * ix;
  const float* pj = A.poses + 7 * jx;
  float q[4];
  relative_pose(pi, pi + 3, pj, pj + 3, g.t, q);
  // quat_rotate's I + 2 w [v] + 2 [v]^2, one rounding an entry
  const double x = q[0], y = q[1], z = q[2], w = q[3];
  g.R[0] = (float)(1.0 - 2.0 * (y * y + z * z));
  g.R[1] = (float)(2.0 * (x * y - w * z));
  g.R[2] = (float)(2.0 * (x * z + w * y));
  g.R[3] = (float)(2.0 * (x * y + w * z));
  g.R[4] = (float)(1.0 - 2.0 * (x * x + z * z));
  g.R[5] = (float)(2.0 * (y * z - w * x));
  g.R[6] = (float)(2.0 * (x * z - w * y));
  g.R[7] = (float)(2.0 * (y * z + w * x));
  g.R[8] = (float)(1.0 - 2.0 * (x * x + y * y));
  g.e = e;
  g.d = A.disps + ix * HW;
  return g;
}

// proj_trans's terms of NP pixels (k, k + kJdThreads) over n edges, added to C and w; the loads of four
// edges are in flight together.  Bound by instruction issue: the rotation is a matrix, formed once an
// edge.  x and y are divided by the depth (1 to 2 us of a call of 258 edges of 43x77).
template <int NP>
__device__ __forceinline__ void add_edges(const JdArgs& A, const JdEdge* edges, int n, int HW, int k, bool first,
                                          float* Cm, float* wm) {
  const float fx = A.intr[0], fy = A.intr[1], cx = A.intr[2], cy = A.intr[3];
  float X[NP][2], C[NP], w[NP];
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    const int kp = k + p * kJdThreads, vi = kp / A.wd;
    X[p][0] = ((float)(kp - vi * A.wd) - cx) / fx;
    X[p][1] = ((float)vi - cy) / fy;
    C[p] = first ? 0.f : Cm[kp];
    w[p] = first ? 0.f : wm[kp];
  }
  for (int j0 = 0; j0 < n; j0 += 4) {
    float h[4][NP], tu[4][NP], tv[4][NP], gu[4][NP], gv[4][NP];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const JdEdge& g = edges[min(j0 + q, n - 1)];
      const float* trg = A.targets + (int64_t)g.e * 2 * HW;
      const float* wgt = A.weights + (int64_t)g.e * 2 * HW;
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        const int kp = k + p * kJdThreads;
        h[q][p] = g.d[kp];
        tu[q][p] = trg[kp];
        tv[q][p] = trg[HW + kp];
        gu[q][p] = wgt[kp];
        gv[q][p] = wgt[HW + kp];
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (j0 + q >= n) break;
      const JdEdge& g = edges[j0 + q];
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        float Y[3];
#pragma unroll
        for (int r = 0; r < 3; ++r)
          Y[r] = fmaf(g.R[3 * r], X[p][0], fmaf(g.R[3 * r + 1], X[p][1], fmaf(h[q][p], g.t[r], g.R[3 * r + 2])));
        const bool bad = Y[2] < kMinDepth;
        const float d = bad ? 0.f : 1.0f / Y[2];
        const float xp = fx * (Y[0] / Y[2]) + cx, yp = fy * (Y[1] / Y[2]) + cy;
        const float d2 = d * d;
        const float wu = bad ? 0.f : 0.001f * gu[q][p];
        const float wv = bad ? 0.f : 0.001f * gv[q][p];
        const float ru = tu[q][p] - xp, rv = tv[q][p] - yp;
        const float Jzu = fx * d * g.t[0] + fx * (-Y[0] * d2) * g.t[2];
        const float Jzv = fy * d * g.t[1] + fy * (-Y[1] * d2) * g.t[2];
        C[p] += wu * Jzu * Jzu + wv * Jzv * Jzv;
        w[p] += wu * ru * Jzu + wv * rv * Jzv;
      }
    }
  }
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    Cm[k + p * kJdThreads] = C[p];
    wm[k + p * kJdThreads] = w[p];
  }
}

// One exchange of block_sum over the first n of acc, and the ones after it.
template <int n, int off, int N>
__device__ __forceinline__ void warp_halve(double (&acc)[N], int& at, int& have) {
  constexpr int h = (n + 1) / 2;
  const bool up = threadIdx.x & off;
#pragma unroll
  for (int i = 0; i < h; ++i) {
    const double lo = acc[i], hi = h + i < n ? acc[h + i] : 0.0;
    acc[i] = (up ? hi : lo) + __shfl_xor_sync(0xffffffffu, up ? lo : hi, off);
  }
  at += up ? h : 0;
  have = up ? have - h : min(have, h);
  if constexpr (off > 1) warp_halve<h, off / 2>(acc, at, have);
}

// Sums of acc over the CTA into tot[0 .. N).  The warp halves the list at every exchange (a lane keeps
// one half and sends the other), 20 exchanges of doubles for 18 sums where five rounds of all are 90.
template <int N>
__device__ __forceinline__ void block_sum(double (&acc)[N], double (*red)[N], double* tot) {
  const int warp = threadIdx.x >> 5;
  int at = 0, have = N;   // this lane's run of the list: start and entries that are not padding
  warp_halve<N, 16>(acc, at, have);
  if (have > 0) red[warp][at] = acc[0];
  __syncthreads();
  if (threadIdx.x < N) {
    double s = 0.0;
    for (int q = 0; q < kJdWarps; ++q) s += red[q][threadIdx.x];
    tot[threadIdx.x] = s;
  }
  __syncthreads();
}

// S + diag(ep + lm Hd) = L L^T in place and x = S^-1 v by one warp, a lane for each row and parity of the
// column; the diagonal of S ends as 1 / L_kk, so that one reciprocal square root is all that a step
// waits for.  Loops stay rolled: each runs once a launch, and fetching unrolled code took longer
// than the arithmetic (4 unknowns: 14k cycles against 5.7k).  False when a pivot is not positive.
__device__ __forceinline__ bool warp_solve(int D, double (*S)[kJdMaxD + 1], const double* Hd, double v, double& x) {
  const int lane = threadIdx.x & 31, row = lane & 15, odd = lane >> 4;
  if (lane < D) S[lane][lane] += kJdEp + kJdLm * Hd[lane];
  __syncwarp();
#pragma unroll 1
  for (int k = 0; k < D; ++k) {
    const double piv = S[k][k];
    if (!(piv > 0.0)) return false;
    const double r = rsqrt(piv);
    const double lk = row > k && row < D ? S[row][k] * r : 0.0;
    const double y = __shfl_sync(0xffffffffu, v, k) * r;
    v = lane == k ? y : lane > k && lane < D ? v - lk * y : v;
    __syncwarp();
    if (!odd && row < D && row >= k) S[row][k] = row == k ? r : lk;
    __syncwarp();
#pragma unroll 1
    for (int l = k + 1 + odd; l < D; l += 2)
      if (row >= l && row < D) S[row][l] -= lk * S[l][k];
    __syncwarp();
  }
#pragma unroll 1
  for (int k = D - 1; k >= 0; --k) {
    const double y = __shfl_sync(0xffffffffu, v, k) * S[k][k];
    v = lane == k ? y : lane < k ? v - S[k][lane] * y : v;
  }
  x = v;
  return true;
}

// kRanks: CTAs of a block; kEdges: C and w are summed here, else they are read
template <int kRanks, bool kEdges>
__global__ void __cluster_dims__(kRanks, 1, 1) __launch_bounds__(kJdThreads, 2)
jdsa_step_kernel(const JdArgs A) {
  extern __shared__ float jd_axes[];   // gy [ht] then gx [wd]
  __shared__ double red[kJdWarps][kJdSums];
  __shared__ double part[kJdMaxCells * kJdSums];   // this CTA's sums, read by the whole cluster
  __shared__ double tot[kJdMaxCells * kJdSums];
  __shared__ double S[kJdMaxD][kJdMaxD + 1];
  __shared__ double Li[kJdMaxD][kJdMaxD + 1];
  __shared__ double Hd[kJdMaxD], v[kJdMaxD];
  __shared__ float dso[kJdMaxD];
  __shared__ float Si[kJdMaxD][kJdMaxD + 1];
  __shared__ float sc_r[kJdMaxD], sc_s[kJdMaxD];
  __shared__ JdEdge edges[kEdges ? kJdBatch : 1];
  __shared__ int list[kEdges ? kJdBatch + kJdThreads : 1];
  __shared__ int found[kJdWarps];
  __shared__ int bad, failed;
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int HW = A.ht * A.wd, D = A.hs * A.ws, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = (int)cluster.block_rank();
  const int b = blockIdx.x / kRanks;
  // an equal run of pixels for each CTA, in whole warps
  const int run = (HW / kRanks + 32) / 32 * 32, k0 = rank * run + tid, kend = min(HW, (rank + 1) * run);
  if (b >= A.M) {
    // frames of the window that are not source frames: the where / clamp only
    const int step = gridDim.x / kRanks - A.M;
    for (int64_t f = b - A.M; f < A.num_disps; f += step) {
      if (find_sorted(A.kx, A.M, f) >= 0) continue;
      const float* src = A.disps + f * HW;
      float* dst = A.out + f * HW;
      for (int k = k0; k < kend; k += kJdThreads) dst[k] = jd_clean(src[k]);
    }
    return;
  }
  // every CTA of a cluster comes to the same verdict here, so none waits for one that left
  const int64_t fr = A.kx[b], want = A.kx[0] + b;
  const int ms = fr == want ? b : find_sorted(A.kx, A.M, want);   // source of block b's prior terms
  const int64_t fs = ms >= 0 ? A.kx[ms] : fr;
  if (tid == 0) {
    bad = fr < 0 || fr >= A.num_disps || fr >= A.num_prior || fr >= A.num_scales || (b > 0 && A.kx[b - 1] >= fr) ||
          fs < 0 || fs >= A.num_disps || fs >= A.num_prior || fs >= A.num_scales;
    failed = 0;
  }
  float* gy = jd_axes;
  float* gx = jd_axes + A.ht;
  for (int i = tid; i < A.ht; i += kJdThreads) gy[i] = A.gy[i];
  for (int j = tid; j < A.wd; j += kJdThreads) gx[j] = A.gx[j];
  if (tid < D) {
    Hd[tid] = 0.0;
    v[tid] = 0.0;
  }
  for (int e = tid; e < kJdMaxD * kJdMaxD; e += kJdThreads) S[e / kJdMaxD][e % kJdMaxD] = 0.0;
  __syncthreads();
  // every grid coordinate needs its 2x2 cell inside the scale grid (bi_inter's bound)
  for (int i = tid; i < A.ht + A.wd; i += kJdThreads) {
    const float c = floorf(i < A.ht ? gy[i] : gx[i - A.ht]);
    const int n = i < A.ht ? A.hs : A.ws;
    if (!(c >= 0.f && c + 1.f < (float)n)) bad = 1;
  }
  __syncthreads();
  if (bad) {
    if (tid == 0) atomicOr(A.info, HS2_DEV_BAD_INDEX);
    return;
  }
  if (tid < D) {
    sc_r[tid] = A.dscales[fr * D + tid];
    sc_s[tid] = A.dscales[fs * D + tid];
  }

  // ---- C and w of this thread's pixels: the edges of slot b in their order
  float* Cm = A.C + (int64_t)b * HW;
  float* wm = A.w + (int64_t)b * HW;
  const int E = kEdges ? (int)A.num_edges : 0;
  int num = 0;         // edges in `list`
  bool first = true;
  for (int base = 0; base < E; base += kJdThreads) {
    const int e = base + tid;
    const int64_t m = e < E ? A.slot[e] : b + 1;
    if (e < E && (m < 0 || m >= A.M)) atomicOr(A.info, HS2_DEV_BAD_INDEX);
    const unsigned mine = __ballot_sync(0xffffffffu, m == b);
    if (lane == 0) found[warp] = __popc(mine);
    __syncthreads();
    int at = num;
    for (int q = 0; q < kJdWarps; ++q) {
      if (q == warp && m == b) list[at + __popc(mine & ((1u << lane) - 1))] = e;
      at += found[q];
    }
    num = at;
    __syncthreads();
    if (num <= kJdBatch && base + kJdThreads < E) continue;
    for (int s = 0; s < num; s += kJdBatch) {
      const int n = min(kJdBatch, num - s);
      if (tid < n) edges[tid] = load_edge(A, list[s + tid], fr, HW);
      __syncthreads();
      int k = k0;
      for (; k + kJdThreads < kend; k += 2 * kJdThreads) add_edges<2>(A, edges, n, HW, k, first, Cm, wm);
      if (k < kend) add_edges<1>(A, edges, n, HW, k, first, Cm, wm);
      first = false;
      __syncthreads();
    }
    num = 0;
  }
  if (kEdges && first)
    for (int k = k0; k < kend; k += kJdThreads) Cm[k] = wm[k] = 0.f;
  __syncthreads();   // sc_r, sc_s

  const bool has_src = ms >= 0;
  const float alpha = A.alpha;
  // ---- pass 1: the block's Schur complement and right-hand side, cell by cell
  const int cells = (A.hs - 1) * (A.ws - 1);
  for (int cell = 0; cell < cells; ++cell) {
    const int cy = cell / (A.ws - 1), cx = cell - cy * (A.ws - 1);
    double acc[kJdSums];
#pragma unroll
    for (int i = 0; i < kJdSums; ++i) acc[i] = 0.0;
    if (has_src) {
      for (int k = k0; k < kend; k += kJdThreads) {
        const int i = k / A.wd, j = k - i * A.wd;
        if ((int)floorf(gy[i]) != cy || (int)floorf(gx[j]) != cx) continue;
        const Cell c = make_cell(gx[j], gy[i], cx, cy, A.ws);
        const RowTerms r = row_terms(A, b, fr, HW, k, sc_r, c);
        const int64_t sk = fs * HW + k;
        const float ps = A.prior[sk];
        const float a = ps > 0.f ? ps : 0.f;
        const float rds = A.disps[sk] - ps * interp(sc_s, c);
        const double ca = (double)(alpha * a * a * (1.0f - alpha * r.Q));
        const double ha = (double)(alpha * a * a);
        const double va = (double)(alpha * a * (rds + r.Q * r.wq));
        int q = 0;
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
#pragma unroll
          for (int ll = kk; ll < 4; ++ll) acc[q++] += ca * c.wt[kk] * c.wt[ll];
        }
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          acc[10 + kk] += ha * c.wt[kk] * c.wt[kk];
          acc[14 + kk] += va * c.wt[kk];
        }
      }
    }
    block_sum<kJdSums>(acc, red, part + cell * kJdSums);
  }
  // the cluster's sums, added in the order of its CTAs by each of them
  cluster.sync();
  for (int i = tid; i < cells * kJdSums; i += kJdThreads) {
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < kRanks; ++q) s += cluster.map_shared_rank(part, q)[i];
    tot[i] = s;
  }
  auto read = cluster.barrier_arrive();   // waited for before this CTA's shared memory goes away
  __syncthreads();

  // ---- damped D x D solve in FP64 by the first warp
  if (warp == 0) {
    for (int cell = 0; cell < cells; ++cell) {
      if (lane < kJdSums) {
        const int cy = cell / (A.ws - 1), p0 = cy * A.ws + cell - cy * (A.ws - 1);
        const int pos[4] = {p0, p0 + A.ws, p0 + 1, p0 + A.ws + 1};
        const double t = tot[cell * kJdSums + lane];
        if (lane < 10) {
          int kk = 0, q = lane;
          while (q >= 4 - kk) { q -= 4 - kk; ++kk; }
          const int ll = kk + q;
          S[pos[kk]][pos[ll]] += t;
          if (ll != kk) S[pos[ll]][pos[kk]] += t;
        } else if (lane < 14) {
          Hd[pos[lane - 10]] += t;
        } else {
          v[pos[lane - 14]] += t;
        }
      }
      __syncwarp();
    }
    double x = 0.0;
    const bool ok = warp_solve(D, S, Hd, lane < D ? v[lane] : 0.0, x);
    if (lane < D) {
      dso[lane] = ok ? (float)x : 0.f;
      if (rank == 0) A.dso[(int64_t)b * D + lane] = dso[lane];
    }
    if (!ok && lane == 0) {
      failed = 1;
      atomicOr(A.info, HS2_DEV_NOT_PD);
    }
    // columns of L^-1 by forward substitution (lane k: L x = e_k)
    if (A.dzcov && ok && lane < D) {
#pragma unroll 1
      for (int i = 0; i < D; ++i) {
        double t = i == lane ? 1.0 : 0.0;
#pragma unroll 1
        for (int m = lane; m < i; ++m) t -= S[i][m] * Li[m][lane];
        Li[i][lane] = i < lane ? 0.0 : t * S[i][i];
      }
    }
  }
  __syncthreads();
  if (A.dzcov) {
    // S^-1 = L^-T L^-1
    for (int e = tid; e < D * D; e += kJdThreads) {
      const int k = e / D, l = e - k * D;
      double s = 0.0;
      if (!failed)
        for (int m = max(k, l); m < D; ++m) s += Li[m][k] * Li[m][l];
      Si[k][l] = (float)s;
    }
    __syncthreads();
  }

  // ---- pass 2: depth update, clean-up and covariance of this thread's pixels of frame fr
  float* outr = A.out + fr * HW;
  float* cov = A.dzcov ? A.dzcov + (int64_t)b * HW : nullptr;
  for (int k = k0; k < kend; k += kJdThreads) {
    const int i = k / A.wd, j = k - i * A.wd;
    const int cy = (int)floorf(gy[i]), cx = (int)floorf(gx[j]);
    const Cell c = make_cell(gx[j], gy[i], cx, cy, A.ws);
    const RowTerms r = row_terms(A, b, fr, HW, k, sc_r, c);
    float a = 0.f;
    if (has_src) {
      const float ps = A.prior[fs * HW + k];
      a = ps > 0.f ? ps : 0.f;
    }
    const float dot = c.wt[0] * dso[c.pos[0]] + c.wt[1] * dso[c.pos[1]] + c.wt[2] * dso[c.pos[2]] +
                      c.wt[3] * dso[c.pos[3]];
    const float dz = r.Q * (r.wq + alpha * a * dot);
    outr[k] = jd_clean(r.d + dz);
    if (cov) {
      float quad = 0.f;
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
#pragma unroll
        for (int ll = 0; ll < 4; ++ll) quad += c.wt[kk] * c.wt[ll] * Si[c.pos[kk]][c.pos[ll]];
      }
      const float e = alpha * a * r.Q;
      cov[k] = e * e * quad + r.Q;
    }
  }
  cluster.barrier_wait(std::move(read));
}

// kx, slot and the number of distinct frames from a bitmap over the frames.
__global__ void __launch_bounds__(kJdKeyThreads)
jdsa_keys_kernel(const int64_t* __restrict__ ii, int E, int frames, int M, int64_t* __restrict__ kx,
                 int64_t* __restrict__ slot, int32_t* __restrict__ count) {
  constexpr int kWords = kJdKeyFrames / 32, kPer = kWords / kJdKeyThreads;
  __shared__ unsigned bits[kWords];
  __shared__ int before[kWords];   // distinct frames ahead of the word
  __shared__ int sums[kJdKeyThreads / 32];
  __shared__ int outside;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < kWords; i += kJdKeyThreads) bits[i] = 0;
  if (tid == 0) outside = 0;
  __syncthreads();
  for (int e = tid; e < E; e += kJdKeyThreads) {
    const int64_t f = ii[e];
    if (f >= 0 && f < frames) atomicOr(&bits[f >> 5], 1u << (f & 31));
    else outside = 1;
  }
  __syncthreads();
  int n = 0;
#pragma unroll
  for (int i = 0; i < kPer; ++i) n += __popc(bits[tid * kPer + i]);
  int scan = n;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, scan, off);
    if (lane >= off) scan += up;
  }
  if (lane == 31) sums[warp] = scan;
  __syncthreads();
  int at = scan - n, total = 0;
  for (int q = 0; q < kJdKeyThreads / 32; ++q) {
    if (q < warp) at += sums[q];
    total += sums[q];
  }
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int word = tid * kPer + i;
    before[word] = at;
    for (unsigned left = bits[word]; left; left &= left - 1, ++at)
      if (at < M) kx[at] = word * 32 + __ffs(left) - 1;
  }
  __syncthreads();
  for (int i = total + tid; i < M; i += kJdKeyThreads) kx[i] = -1;
  for (int e = tid; e < E; e += kJdKeyThreads) {
    const int64_t f = ii[e];
    int64_t at_f = -1;
    if (f >= 0 && f < frames) at_f = before[f >> 5] + __popc(bits[f >> 5] & ((1u << (f & 31)) - 1));
    slot[e] = at_f;
  }
  if (tid == 0) *count = outside ? -1 : total;
}

__global__ void __launch_bounds__(kJdThreads)
jdsa_scales_kernel(float* __restrict__ dscales, int D, const int64_t* __restrict__ kx, int M,
                   const float* __restrict__ dso, const int32_t* __restrict__ info) {
  if (*info & (HS2_DEV_BAD_INDEX | HS2_DEV_NOT_PD)) return;
  for (int t = blockIdx.x * kJdThreads + threadIdx.x; t < M * D; t += gridDim.x * kJdThreads) {
    const int b = t / D, k = t - b * D;
    dscales[kx[b] * D + k] += dso[t];
  }
}

}  // namespace
}  // namespace hs2

extern "C" int hs2_jdsa_keys(const int64_t* ii, int64_t num_edges, int64_t num_frames, int64_t num_kx, int64_t* kx,
                             int64_t* slot, int32_t* count, hs2_stream_t stream) {
  using namespace hs2;
  if (num_edges <= 0 || num_edges > 0x7fffffff || num_frames <= 0 || num_frames > kJdKeyFrames || num_kx <= 0 ||
      num_kx > num_edges) {
    set_error("jdsa_keys: bad counts (edges %lld, frames %lld of at most %d, source frames %lld)",
              (long long)num_edges, (long long)num_frames, kJdKeyFrames, (long long)num_kx);
    return HS2_ERR_INVALID;
  }
  if (!ii || !kx || !slot || !count) {
    set_error("jdsa_keys: a required pointer is null");
    return HS2_ERR_INVALID;
  }
  int rc = bind_device(kx);
  if (rc) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  HS2_PROF("jdsa_keys", s);
  jdsa_keys_kernel<<<1, kJdKeyThreads, 0, s>>>(ii, (int)num_edges, (int)num_frames, (int)num_kx, kx, slot, count);
  HS2_LAUNCH_CHECK("jdsa_keys_kernel");
  return HS2_OK;
}

extern "C" int hs2_jdsa(const float* poses, int64_t num_poses, const float* disps, int64_t num_disps, int ht, int wd,
                        const float* intrinsics, const float* targets, const float* weights, const float* eta,
                        const float* disps_prior, int64_t num_prior, float* dscales, int64_t num_scales, int hs,
                        int ws, const float* grid_y, const float* grid_x, const int64_t* ii, const int64_t* jj,
                        const int64_t* slot, int64_t num_edges, const int64_t* kx, int64_t num_kx, float alpha,
                        float* C, float* w, float* dso, float* disps_out, float* dzcov, int32_t* info,
                        hs2_stream_t stream) {
  using namespace hs2;
  if (num_poses < 0 || num_disps <= 0 || num_disps > 0x7fffffff - 65536 || ht <= 0 || wd <= 0 ||
      ht > kJdMaxAxis || wd > kJdMaxAxis || (int64_t)ht * wd > (1 << 30) || num_prior < 0 || num_scales < 0 ||
      hs < 2 || ws < 2 || hs * ws > kJdMaxD || num_edges < 0 || num_edges > 0x7fffffff) {
    set_error("jdsa: bad sizes (num_disps %lld, ht %d, wd %d, hs %d, ws %d, edges %lld; needs 2 <= hs, ws, "
              "hs*ws <= %d, ht, wd <= %d)", (long long)num_disps, ht, wd, hs, ws, (long long)num_edges, kJdMaxD,
              kJdMaxAxis);
    return HS2_ERR_INVALID;
  }
  if (num_kx <= 0 || num_kx > 65535 || num_kx > num_edges) {
    set_error("jdsa: %lld source frames for %lld edges (the reference indexes kx[0]: at least one edge)",
              (long long)num_kx, (long long)num_edges);
    return HS2_ERR_INVALID;
  }
  if (!grid_y || !grid_x || !kx || !C || !w || !dso || !disps_out || !info) {
    set_error("jdsa: a required pointer is null");
    return HS2_ERR_INVALID;
  }
  int rc = bind_device(disps_out);
  if (rc) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  HS2_CUDA(cudaMemsetAsync(info, 0, sizeof(int32_t), s));
  JdArgs A;
  A.poses = poses;
  A.num_poses = num_poses;
  A.intr = intrinsics;
  A.targets = targets;
  A.weights = weights;
  A.ii = ii;
  A.jj = jj;
  A.slot = slot;
  A.num_edges = num_edges;
  A.disps = disps;
  A.num_disps = num_disps;
  A.ht = ht;
  A.wd = wd;
  A.C = C;
  A.w = w;
  A.eta = eta;
  A.prior = disps_prior;
  A.num_prior = num_prior;
  A.dscales = dscales;
  A.num_scales = num_scales;
  A.hs = hs;
  A.ws = ws;
  A.gy = grid_y;
  A.gx = grid_x;
  A.kx = kx;
  A.M = (int)num_kx;
  A.alpha = alpha;
  A.dso = dso;
  A.out = disps_out;
  A.dzcov = dzcov;
  A.info = info;
  const size_t smem = sizeof(float) * (size_t)(ht + wd);
  const bool fused = num_kx <= kJdFusedBlocks;
  if (!fused && (rc = hs2_proj_trans(poses, num_poses, disps, num_disps, ht, wd, intrinsics, targets, weights, ii, jj,
                                     slot, num_edges, num_kx, C, w, info, stream)))
    return rc;
  // every frame that is not a source frame is one of num_disps - M
  const unsigned copies = (unsigned)std::min<int64_t>(std::max<int64_t>(num_disps - num_kx, 0), kJdCopyClusters);
  HS2_PROF("jdsa_step", s);
  const unsigned clusters = (unsigned)num_kx + copies;
  if (fused)
    jdsa_step_kernel<kJdCluster, true><<<clusters * kJdCluster, kJdThreads, smem, s>>>(A);
  else
    jdsa_step_kernel<kJdPlainCluster, false><<<clusters * kJdPlainCluster, kJdThreads, smem, s>>>(A);
  HS2_LAUNCH_CHECK("jdsa_step_kernel");
  const int D = hs * ws;
  HS2_PROF("jdsa_scales", s);
  jdsa_scales_kernel<<<(unsigned)std::min<int64_t>(64, (num_kx * D + kJdThreads - 1) / kJdThreads), kJdThreads, 0,
                       s>>>(dscales, D, kx, (int)num_kx, dso, info);
  HS2_LAUNCH_CHECK("jdsa_scales_kernel");
  return HS2_OK;
}
