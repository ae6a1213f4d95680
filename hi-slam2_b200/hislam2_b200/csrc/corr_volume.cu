// All-pairs correlation volume and its 4-level pooling pyramid on the tensor cores.
//
// Replaces the caller-side construction of HI-SLAM2's CorrBlock
// (hislam2/modules/corr.py:29-38 and :63-71):
//   corr[e, y1, x1, y2, x2] = sum_c (fmap1[e, c, y1, x1] / 4) (fmap2[e, c, y2, x2] / 4)
//   level 0 = corr (layout [E, H, W, H, W]),
//   level l = avg_pool2d(level l-1, 2, stride 2) over (y2, x2) (floor sizes),
// i.e. torch.matmul((f1/4)^T, f2/4) followed by three avg_pool2d calls, with the
// same rounding: every level is rounded to the volume's type and pooled from the
// rounded values of the level above, summing the 2x2 window in float in the order
// (y,x), (y,x+1), (y+1,x), (y+1,x+1) and dividing by 4.
//
// Two kernels:
//   corr_pack      fmaps [K, 128, H, W] -> K-major operand rows [K, H*W, 128]
//                  (x 0.25, which is exact; or, for the FP8 form, e4m3 values with one
//                  scale per pixel: q = e4m3(f/4 / s), s = max_c |f/4| / 448);
//   corr_volume    persistent (two CTAs per SM), one work unit = (edge, 128 source
//                  pixels, a run of target image rows that starts at a multiple of 8).
//                  Warp 0 streams the unit's A tile (128 source pixels x 128 channels)
//                  and, per target image row, the B tile (a box of RW = round_up(W, 16)
//                  pixels; pixels past the frame read as zero) with 3-D TMA boxes (128B
//                  swizzle) into a 2-stage ring; warp 1 issues tcgen05.mma (kind::f16
//                  for F16/BF16, kind::f8f6f4 for E4M3; M = 128, N = RW, accumulator
//                  F32) into a ring of TMEM column ranges, one per image row; warps 2-5
//                  (one per TMEM lane quarter, lane = source pixel) drain it for level
//                  0, warps 6-9 for the pooled levels.
// Epilogue: a lane owns a source pixel.  Each level of a source pixel is one contiguous run
// of the output that grows with the image rows, so per image row and level a lane
// appends its new elements, 16 accumulator columns at a time, to its row of a per-warp
// staging buffer at the run's 16-byte phase in global memory; the warp then writes all
// full 16-byte chunks (neighbouring lanes, neighbouring chunks) and each lane keeps its
// partial chunk in registers for the next append.  A level may start at any element: the chunks
// are those of its address, not of its element indices.  Level 1 reads the two image rows'
// accumulators again from TMEM and pools the rounded values; the rows above of levels 1
// and 2 wait in shared memory.  No barrier spans the epilogue warps, single elements are
// written only at the ends of a unit's runs, and everything runs in short loops: the
// same epilogue unrolled over the columns missed the instruction cache and took 3.2 ms.
// The volume is never re-read: the HBM traffic is the pyramid's writes plus the
// operand reads (L2-resident: one frame's operand rows are 848 KB at 43x77).
// Bound by instruction issue (IPC 1.8 per SM, 20% of the stalls on instruction fetch): the
// DRAM floor is a third.  48 edges of 43x77, FP16, four levels: 0.68 ms, and 84 edges of
// 48x64: 0.79 ms, against 1.40 and 1.94 ms for sixteen epilogue warps sharing a staging tile
// between barriers (pooling from shared memory, element-wise run ends on every tile).
//
// Limits: 128 channels, W <= 96, H*W < 2^31 / 128.  Output element offsets are 64-bit.
#include <cuda_fp8.h>

#include <algorithm>

#include "profile.cuh"
#include "tc.cuh"

namespace hs2 {

namespace {

constexpr int kCvC = 128;          // feature channels (K of the contraction)
constexpr int kCvMaxW = 96;        // widest image row a B box holds
constexpr int kCvEpiWarps = 8;     // per TMEM lane quarter one for level 0, one for the pooled levels
constexpr int kCvThreads = 32 * (2 + kCvEpiWarps);   // TMA, MMA, epilogue
constexpr int kCvTmemCols = 256;
constexpr int kCvMaxRegions = 4;   // image rows held in TMEM
constexpr uint32_t kCvMinSmem = 77 * 1024, kCvPairSmem = 113 * 1024;   // two CTAs per SM (they fill TMEM)
constexpr uint32_t kCvASub = 128 * 128;   // one 128-row x 128-byte swizzled sub-tile

// operand forms: F16 / BF16 (kind::f16), E4M3 with per-pixel scales (kind::f8f6f4)
constexpr int kF16 = 0, kBF16 = 1, kE4M3 = 2;
template <int P> struct Prec;
template <> struct Prec<kF16> {
  static constexpr int kEsize = 2, kSub = 2, kFmt = 0;
};
template <> struct Prec<kBF16> {
  static constexpr int kEsize = 2, kSub = 2, kFmt = 1;
};
template <> struct Prec<kE4M3> {
  static constexpr int kEsize = 1, kSub = 1, kFmt = 0;
};

struct CvGeom {
  int H, W, HW, RW;
  int H1, W1, H2, W2, H3, W3;      // pooled level sizes
  int levels, mtiles, splits, split_rows;
  int64_t E;
  int stages, regions;             // B tiles in flight, accumulators in TMEM
  // 16-byte chunks per lane (odd): staging rows of level 0 and of the pooled levels, level-1 and
  // level-2 row above
  int chunks, chunks_p, chunks1, chunks2;
  uint32_t sub_b;                  // bytes of one B sub-tile (RW rows x 128 B)
  uint32_t off_b, off_stg, off_stp, off_p1, off_p2, off_bar, smem;
};

CvGeom cv_geom(int H, int W, int64_t E, int levels, int esub) {
  CvGeom g;
  g.H = H;
  g.W = W;
  g.HW = H * W;
  g.RW = (W + 15) & ~15;
  g.H1 = H / 2, g.W1 = W / 2, g.H2 = g.H1 / 2, g.W2 = g.W1 / 2, g.H3 = g.H2 / 2, g.W3 = g.W2 / 2;
  g.levels = levels;
  g.mtiles = (g.HW + 127) / 128;
  g.E = E;
  // image rows per unit: whole frames unless that leaves the last of few waves mostly empty;
  // runs of a multiple of 8 rows keep the pooled levels inside a unit
  const int groups = (H + 7) / 8;
  const int64_t whole = std::max<int64_t>(1, E * g.mtiles);
  const int want = (int)std::min<int64_t>(groups, std::max<int64_t>(1, (8 * 2 * kNumSMs + whole - 1) / whole));
  g.split_rows = 8 * ((groups + want - 1) / want);
  g.splits = (H + g.split_rows - 1) / g.split_rows;
  g.sub_b = (uint32_t)(g.RW * 128);
  g.regions = std::min(kCvMaxRegions, kCvTmemCols / g.RW);
  g.chunks = (((7 + W) >> 3) + 1) | 1;
  g.chunks_p = (((7 + g.W1) >> 3) + 1) | 1;
  g.chunks1 = (g.RW / 16) | 1;
  g.chunks2 = ((g.RW + 31) / 32) | 1;
  g.off_b = (uint32_t)esub * kCvASub;
  // two B tiles in flight and two CTAs per SM; at W > 64 one B tile (the ring of accumulators covers its
  // load), at W > 80 two B tiles in one CTA
  for (int n : {2, 1, 2}) {
    g.stages = n;
    g.off_stg = g.off_b + g.stages * esub * g.sub_b;
    g.off_stp = g.off_stg + 4 * (32u * g.chunks * 16 + 64);
    g.off_p1 = g.off_stp + 4 * (32u * g.chunks_p * 16 + 64);
    g.off_p2 = g.off_p1 + 128u * 16 * g.chunks1;
    g.off_bar = g.off_p2 + 128u * 16 * g.chunks2;
    g.smem = std::max(kCvMinSmem, g.off_bar + 256 + 1024);   // barriers, flags, TMEM slot; 1 KB alignment slack
    if (g.smem <= kCvPairSmem) break;
  }
  return g;
}

template <typename T> __device__ __forceinline__ uint16_t bits16(T v);
template <> __device__ __forceinline__ uint16_t bits16<__half>(__half v) { return __half_as_ushort(v); }
template <> __device__ __forceinline__ uint16_t bits16<__nv_bfloat16>(__nv_bfloat16 v) {
  return __bfloat16_as_ushort(v);
}
template <typename T> __device__ __forceinline__ T from_bits16(uint16_t b);
template <> __device__ __forceinline__ __half from_bits16<__half>(uint16_t b) { return __ushort_as_half(b); }
template <> __device__ __forceinline__ __nv_bfloat16 from_bits16<__nv_bfloat16>(uint16_t b) {
  return __ushort_as_bfloat16(b);
}

// Bounded wait that ignores the abort flag: used on the way out to let copies and
// MMAs that were already issued land before the CTA releases its memory.
__device__ __forceinline__ void drain_wait(uint32_t bar, uint32_t parity) {
  for (unsigned i = 0; i < tc::kSpin && !tc::mbar_test(bar, parity); ++i) {
  }
}

// Two floats rounded to T, the first in the low half.
template <typename T> __device__ __forceinline__ uint32_t pack2(float lo, float hi);
template <> __device__ __forceinline__ uint32_t pack2<__half>(float lo, float hi) {
  const __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}
template <> __device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}
template <typename T> __device__ __forceinline__ float2 unpack2(uint32_t w) {
  return make_float2(to_f<T>(from_bits16<T>((uint16_t)w)), to_f<T>(from_bits16<T>((uint16_t)(w >> 16))));
}

// 2x2 average of the rounded pairs (y, x), (y, x+1) and (y+1, x), (y+1, x+1), in avg_pool2d's order.
template <typename T>
__device__ __forceinline__ float pool4(uint32_t top, uint32_t bottom) {
  const float2 a = unpack2<T>(top), b = unpack2<T>(bottom);
  // the + 0 turns a sum of negative zeros into the 0 that avg_pool2d's sum from 0 gives
  return fmaf(a.x + a.y + b.x + b.y, 0.25f, 0.f);
}

// How the warp's lanes share a flush of up to `per` full chunks a row: lane = (row of a group,
// chunk); the chunk stays, the rows step by whole groups.
struct CvShare {
  int group, r0, c;
  __device__ explicit CvShare(int n) {
    const int per = (7 + n) >> 3, lane = threadIdx.x & 31;
    group = per > 0 ? 32 / per : 32;
    r0 = per > 0 ? lane / per : 0;
    c = lane - r0 * per;
    if (per == 0 || r0 >= group) r0 = 32;             // idle
  }
};

// Writes the warp's full chunks after an append of n elements.  Row r of the warp holds the
// run of source pixel r; its new elements start at out[g0 + r * plane] (out on a 16-byte boundary),
// `since` elements after the unit's part of the run began.  rows: live rows of the warp; done: the unit's last append.
// Returns the lane's partial chunk.
// One copy for all levels: inlined everywhere, the epilogue's loops outgrow the instruction cache.
__device__ __noinline__ uint4 run_flush(const CvShare sh, uint16_t* __restrict__ out, int64_t g0, int plane, int n,
                                        int since, bool done, int rows, int chunks, const uint8_t* stg) {
  const int lane = threadIdx.x & 31;
  __syncwarp();
  const int ph0 = (int)(g0 & 7);
  uint16_t* base = out + (g0 - ph0);
  // a chunk that also holds elements before the unit's part of the run (chunk 0 at a phase beyond
  // `since`) is left to its lane
  const int lim = sh.c == 0 ? since : 8, step = sh.group * plane;
  int rel = ph0 + sh.r0 * plane;
#pragma unroll 2
  for (int r = sh.r0; r < rows; r += sh.group, rel += step) {
    const int off = rel & 7;
    if (8 * sh.c + 8 <= off + n && off <= lim) {
      const uint4 v = *reinterpret_cast<const uint4*>(stg + 16 * (r * chunks + (r >> 3) + sh.c));
      *reinterpret_cast<uint4*>(base + (rel - off + 8 * sh.c)) = v;
    }
  }
  rel = ph0 + lane * plane;
  const int off = rel & 7, total = off + n;
  const uint8_t* row = stg + 16 * (lane * chunks + (lane >> 3));
  if ((since < 8 || done) && lane < rows) {           // the ends of the unit's part of the run
    const uint16_t* el = reinterpret_cast<const uint16_t*>(row);
    uint16_t* dst = base + (rel - off);
    const int head = off > since ? off - since : 0;   // elements of chunk 0 that are not the unit's
    if (head && total >= 8)
      for (int i = head; i < 8; ++i) dst[i] = el[i];
    if (done)
      for (int i = max(total & ~7, head); i < total; ++i) dst[i] = el[i];
  }
  const uint4 tail = *reinterpret_cast<const uint4*>(row + 16 * (total >> 3));
  __syncwarp();
  return tail;
}

// A lane's append to its staging row, word by word.  At an odd phase every stored word joins
// the halves of neighbouring pairs: one byte permute, whose selector is the lane's.
struct CvAppend {
  uint32_t* dst;
  uint32_t prev, sel;
  int left;                                           // words to store
  // n elements at phase off, after the run's partial chunk
  __device__ CvAppend(uint8_t* row, const uint4& tail, int off, int n) {
    *reinterpret_cast<uint4*>(row) = tail;
    const int odd = off & 1;
    prev = odd ? (uint32_t)reinterpret_cast<const uint16_t*>(row)[off - 1] << 16 : 0u;
    sel = odd ? 0x5432u : 0x7654u;
    dst = reinterpret_cast<uint32_t*>(row) + (off >> 1);
    left = (n + odd + 1) >> 1;
  }
  template <int K>
  __device__ __forceinline__ void put(const uint32_t (&w)[K]) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      if (k < left) dst[k] = __byte_perm(prev, w[k], sel);
      prev = w[k];
    }
    dst += K;
    left -= K;
  }
  // as put, for words that all belong to the run
  template <int K>
  __device__ __forceinline__ void put_full(const uint32_t (&w)[K]) {
#pragma unroll
    for (int k = 0; k < K; ++k) dst[k] = __byte_perm(k ? w[k - 1] : prev, w[k], sel);
    prev = w[K - 1];
    dst += K;
    left -= K;
  }
  __device__ __forceinline__ void end() {             // an odd phase's last half word
    if (left > 0) *dst = __byte_perm(prev, 0u, sel);
  }
};

}  // namespace

// ----------------------------------------------------------------- pack ---
// fmaps [K, 128, HW] (T) -> rows [K, HW, 128] of the operand type; 64 pixels per CTA.  A thread's 32
// loads go out eight at a time: one by one, behind a bounds test each, they took 64 us for the
// 2 x 48 frames of 43x77 in float16 (81 MB each way, 25 us at the copy rate), now 55.
template <typename T, int P>
__global__ void __launch_bounds__(256) corr_pack_kernel(const T* __restrict__ f, int HW, void* __restrict__ rows,
                                                        float* __restrict__ scale) {
  __shared__ float tile[kCvC][65];
  __shared__ float amax[64];
  const int k = blockIdx.y;
  const int p0 = blockIdx.x * 64;
  const T* src = f + (int64_t)k * kCvC * HW;
  {
    const int p = threadIdx.x & 63, at = min(p0 + p, HW - 1);   // pixels past the frame are not stored
#pragma unroll
    for (int c0 = threadIdx.x >> 6; c0 < kCvC; c0 += 32) {
      T v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = src[(int64_t)(c0 + 4 * i) * HW + at];
#pragma unroll
      for (int i = 0; i < 8; ++i) tile[c0 + 4 * i][p] = to_f<T>(v[i]) * 0.25f;
    }
  }
  __syncthreads();
  if (P == kE4M3) {
    // per-pixel scale: 8 threads per pixel reduce |x| over the 128 channels
    const int p = threadIdx.x >> 2, part = threadIdx.x & 3;
    float m = 0.f;
    for (int c = part; c < kCvC; c += 4) m = fmaxf(m, fabsf(tile[c][p]));
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
    if (part == 0) {
      const float s = m > 0.f ? m / 448.0f : 1.0f;
      amax[p] = s;
      if (p0 + p < HW) scale[(int64_t)k * HW + p0 + p] = s;
    }
    __syncthreads();
    uint8_t* out = static_cast<uint8_t*>(rows) + ((int64_t)k * HW + p0) * kCvC;
    for (int i = threadIdx.x; i < 64 * kCvC / 2; i += 256) {
      const int p = i / (kCvC / 2), c = (i - p * (kCvC / 2)) * 2;
      if (p0 + p >= HW) continue;
      const float inv = 1.0f / amax[p];
      const __nv_fp8x2_storage_t q =
          __nv_cvt_float2_to_fp8x2(make_float2(tile[c][p] * inv, tile[c + 1][p] * inv), __NV_SATFINITE, __NV_E4M3);
      *reinterpret_cast<__nv_fp8x2_storage_t*>(out + (int64_t)p * kCvC + c) = q;
    }
  } else {
    using OpT = typename std::conditional<P == kBF16, __nv_bfloat16, __half>::type;
    OpT* out = static_cast<OpT*>(rows) + ((int64_t)k * HW + p0) * kCvC;
    const int end = min(64, HW - p0) * (kCvC / 2);
#pragma unroll 4
    for (int i = threadIdx.x; i < end; i += 256) {
      const int p = i / (kCvC / 2), c = (i - p * (kCvC / 2)) * 2;
      const uint32_t lo = bits16<OpT>(from_f<OpT>(tile[c][p])), hi = bits16<OpT>(from_f<OpT>(tile[c + 1][p]));
      *reinterpret_cast<uint32_t*>(out + (int64_t)p * kCvC + c) = lo | (hi << 16);
    }
  }
}

// --------------------------------------------------------------- volume ---
// A level's output: the 16-byte boundary at or before its first element, and how many elements before
// it that boundary lies.  Run positions count from the boundary, so a multiple of 8 is aligned.
struct CvOut {
  uint16_t* lvl[4];
  int skew[4];
};

template <int P, typename T>
__global__ void __launch_bounds__(kCvThreads, 2)
corr_volume_kernel(const __grid_constant__ CUtensorMap amap, const __grid_constant__ CUtensorMap bmap,
                   const int64_t* __restrict__ ii, const int64_t* __restrict__ jj, int64_t K1, int64_t K2,
                   const float* __restrict__ s1, const float* __restrict__ s2, const __grid_constant__ CvGeom g,
                   const __grid_constant__ CvOut out,
                   int32_t* __restrict__ info) {
  using PR = Prec<P>;
  extern __shared__ uint8_t cv_raw[];
  const uint32_t raw = tc::smem_u32(cv_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* gb = cv_raw + (base - raw);
  uint64_t* bars = reinterpret_cast<uint64_t*>(gb + g.off_bar);
  // a_full, a_empty, b_full[2], b_empty[2], t_full[4], t_empty[4], mma_done
  const uint32_t bar0 = tc::smem_u32(bars);
  const uint32_t a_full = bar0, a_empty = bar0 + 8;
  const uint32_t b_full = bar0 + 16, b_empty = bar0 + 32, t_full = bar0 + 48, t_empty = bar0 + 80;
  const uint32_t mma_done = bar0 + 112;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gb + g.off_bar + 128);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gb + g.off_bar + 136);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    tc::mbar_init(a_full, 1);
    tc::mbar_init(a_empty, 1);
    for (int s = 0; s < g.stages; ++s) {
      tc::mbar_init(b_full + 8 * s, 1);
      tc::mbar_init(b_empty + 8 * s, 1);
    }
    for (int b = 0; b < g.regions; ++b) {
      tc::mbar_init(t_full + 8 * b, 1);
      tc::mbar_init(t_empty + 8 * b, kCvEpiWarps);
    }
    tc::mbar_init(mma_done, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::smem_u32(tmem_slot)),
                 "r"(kCvTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = *tmem_slot;

  const int64_t units = g.E * g.mtiles * g.splits;
  const uint32_t b_stage = (uint32_t)PR::kSub * g.sub_b;
  const int kbox = 128 / PR::kEsize;                  // elements per 128-byte box row
  // unit u -> edge, first source pixel, image rows [i0, i1)
  auto unit_of = [&](int64_t u, int64_t& e, int& m0, int& i0, int& i1) {
    const int64_t em = u / g.splits;
    i0 = (int)(u - em * g.splits) * g.split_rows;
    i1 = min(g.H, i0 + g.split_rows);
    e = em / g.mtiles;
    m0 = (int)(em - e * g.mtiles) * 128;
  };

  if (warp == 0) {
    // ------------------------------------------------------------- TMA producer
    if (lane == 0) {
      uint32_t gt = 0, ul = 0;
      for (int64_t u = blockIdx.x; u < units; u += gridDim.x) {
        int64_t e;
        int m0, i0, i1;
        unit_of(u, e, m0, i0, i1);
        const int64_t fi = ii[e], fj = jj[e];
        if (fi < 0 || fi >= K1 || fj < 0 || fj >= K2) continue;   // every role skips the unit
        if (ul > 0 && !tc::mbar_wait(a_empty, (ul - 1) & 1, abort_flag)) break;
        ++ul;
        tc::mbar_arrive_tx(a_full, PR::kSub * kCvASub);
        for (int kb = 0; kb < PR::kSub; ++kb)
          tc::tma_load_3d(base + kb * kCvASub, &amap, kb * kbox, m0, (int)fi, a_full);
        bool ok = true;
        for (int i = i0; i < i1; ++i, ++gt) {
          const int s = gt % g.stages;
          if (gt >= g.stages && !tc::mbar_wait(b_empty + 8 * s, ((gt / g.stages) - 1) & 1, abort_flag)) {
            ok = false;
            break;
          }
          tc::mbar_arrive_tx(b_full + 8 * s, (uint32_t)(PR::kSub * g.RW * 128));
          const uint32_t dst = base + g.off_b + s * b_stage;
          for (int kb = 0; kb < PR::kSub; ++kb)
            tc::tma_load_3d(dst + kb * g.sub_b, &bmap, kb * kbox, i * g.W, (int)fj, b_full + 8 * s);
        }
        if (!ok) break;
      }
      // let the copies already issued land before the CTA's shared memory is released
      if (ul > 0) drain_wait(a_full, (ul - 1) & 1);
      for (uint32_t k = gt > (uint32_t)g.stages ? gt - g.stages : 0; k < gt; ++k)
        drain_wait(b_full + 8 * (k % g.stages), (k / g.stages) & 1);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------- MMA issuer
    if (lane == 0) {
      uint32_t gt = 0, ul = 0;
      const uint32_t id = tc::idesc(128, g.RW, PR::kFmt);
      for (int64_t u = blockIdx.x; u < units; u += gridDim.x) {
        int64_t e;
        int m0, i0, i1;
        unit_of(u, e, m0, i0, i1);
        const int64_t fi = ii[e], fj = jj[e];
        if (fi < 0 || fi >= K1 || fj < 0 || fj >= K2) continue;
        if (!tc::mbar_wait(a_full, ul & 1, abort_flag)) break;
        ++ul;
        bool ok = true;
        for (int i = i0; i < i1; ++i, ++gt) {
          const uint32_t s = gt % g.stages, b = gt % g.regions, used = gt / g.regions;
          if (!tc::mbar_wait(b_full + 8 * s, (gt / g.stages) & 1, abort_flag) ||
              (used > 0 && !tc::mbar_wait(t_empty + 8 * b, (used - 1) & 1, abort_flag))) {
            ok = false;
            break;
          }
          tc::fence_after();
          const uint32_t bsrc = base + g.off_b + s * b_stage;
          const uint32_t d = tmem + b * g.RW;
#pragma unroll
          for (int kb = 0; kb < PR::kSub; ++kb)
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
              const uint64_t ad = tc::desc_sw128(base + kb * kCvASub + kk * 32);
              const uint64_t bd = tc::desc_sw128(bsrc + kb * g.sub_b + kk * 32);
              if (P == kE4M3) tc::mma_f8(d, ad, bd, id, (kb | kk) ? 1u : 0u);
              else tc::mma_f16(d, ad, bd, id, (kb | kk) ? 1u : 0u);
            }
          tc::commit(b_empty + 8 * s);
          tc::commit(t_full + 8 * b);
        }
        if (!ok) break;
        tc::commit(a_empty);
      }
      // every MMA issued has completed before TMEM is released
      tc::commit(mma_done);
      drain_wait(mma_done, 0);
    }
  } else {
    // ------------------------------------------------------------- epilogue
    const int q = warp & 3;                  // TMEM lane quarter
    const bool pooled = warp >= 6;           // this warp's levels: 0, or 1 to 3
    const int np = g.RW / 16;                // 16-column pieces of an image row
    const int chunks = pooled ? g.chunks_p : g.chunks;
    uint8_t* stg = gb + (pooled ? g.off_stp : g.off_stg) + q * (32 * chunks * 16 + 64);
    // the skew of one chunk per eight rows spreads the rows of a store over the banks
    uint8_t* row = stg + 16 * (lane * chunks + (lane >> 3));
    const uint32_t tq = tmem + ((uint32_t)(q * 32) << 16);
    uint32_t reg = 0, par = 0;               // the next accumulator row's TMEM range and barrier phase
    const uint32_t last_reg = g.regions - 1;
    auto next_row = [&]() {
      if (reg == last_reg) {
        reg = 0;
        par ^= 1;
      } else {
        ++reg;
      }
    };
    for (int64_t u = blockIdx.x; u < units; u += gridDim.x) {
      int64_t e;
      int m0, i0, i1;
      unit_of(u, e, m0, i0, i1);
      const int64_t fi = ii[e], fj = jj[e];
      if (fi < 0 || fi >= K1 || fj < 0 || fj >= K2) {
        if (tid == 64 && m0 == 0) atomicOr(info, HS2_DEV_BAD_INDEX);
        continue;
      }
      const int64_t px0 = e * g.HW + m0 + 32 * q;                 // the warp's first source pixel
      const int rows = min(32, g.HW - m0 - 32 * q);               // live ones (may be <= 0)
      float sa = 1.f;
      if (P == kE4M3) sa = lane < rows ? s1[fi * g.HW + m0 + 32 * q + lane] : 0.f;
      // waits for the accumulator in TMEM range r (uniform over the warp)
      auto wait_row = [&](uint32_t r, uint32_t ph) -> bool {
        const bool ok = tc::mbar_wait(t_full + 8 * r, ph, abort_flag);
        tc::fence_after();
        return __all_sync(0xffffffffu, ok);
      };
      auto free_row = [&](uint32_t r) {
        if (lane == 0) tc::mbar_arrive(t_empty + 8 * r);
      };
      auto load = [&](uint32_t r, int pc, uint32_t (&v)[16]) { tc::ld16(tq + r * g.RW + 16 * pc, v); };
      // the 16 values of piece pc of image row i, rounded, in 8 words
      auto pack = [&](uint32_t (&v)[16], int i, int pc, uint32_t (&w)[8]) {
        if (P == kE4M3) {
          const float* sc = s2 + fj * g.HW + (int64_t)i * g.W;
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            const int x = 16 * pc + k;
            v[k] = __float_as_uint(__uint_as_float(v[k]) * sa * (x < g.W ? __ldg(sc + x) : 0.f));
          }
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) w[k] = pack2<T>(__uint_as_float(v[2 * k]), __uint_as_float(v[2 * k + 1]));
      };
      bool ok = true;
      if (!pooled) {
        const CvShare sh(g.W);
        uint4 tail = make_uint4(0, 0, 0, 0);
        for (int i = i0; i < i1; ++i) {
          if (!(ok = wait_row(reg, par))) break;
          const int64_t g0 = px0 * g.HW + (int64_t)i * g.W + out.skew[0];
          CvAppend ap(row, tail, ((int)(g0 & 7) + lane * g.HW) & 7, g.W);
          uint32_t v[2][16], w[8];
          load(reg, 0, v[0]);
          int pc = 0;
          for (; pc + 2 < np; pc += 2) {                          // the next piece's load runs under this one's stores
            tc::ld_wait();
            load(reg, pc + 1, v[1]);
            pack(v[0], i, pc, w);
            ap.put_full(w);
            tc::ld_wait();
            load(reg, pc + 2, v[0]);
            pack(v[1], i, pc + 1, w);
            ap.put_full(w);
          }
          tc::ld_wait();
          if (pc + 1 < np) {
            load(reg, pc + 1, v[1]);
            pack(v[0], i, pc, w);
            ap.put_full(w);
            tc::ld_wait();
#pragma unroll
            for (int k = 0; k < 16; ++k) v[0][k] = v[1][k];
            ++pc;
          }
          tc::fence_before();
          __syncwarp();
          free_row(reg);
          pack(v[0], i, pc, w);
          ap.put(w);
          ap.end();
          tail = run_flush(sh, out.lvl[0], g0, g.HW, g.W, (i - i0) * g.W, i == i1 - 1, rows, chunks, stg);
          next_row();
        }
      } else {
        uint8_t* p1 = gb + g.off_p1 + 16 * (32 * q + lane) * g.chunks1;   // per piece: 4 words of level 1, then 2 of level 2
        uint8_t* p2 = gb + g.off_p2 + 16 * (32 * q + lane) * g.chunks2;   // per piece: 2 words of level 2, then 1 of level 3
        const CvShare sh1(g.W1), sh2(g.W2), sh3(g.W3);
        const int HW1 = g.H1 * g.W1, HW2 = g.H2 * g.W2, HW3 = g.H3 * g.W3;
        uint4 tail1 = make_uint4(0, 0, 0, 0), tail2 = tail1, tail3 = tail1;
        for (int i = i0; i < i1; i += 2) {
          const bool two = i + 1 < i1;
          const int j = i >> 1, j2 = i >> 2, j3 = i >> 3;
          const uint32_t ra = reg;
          if (!(ok = wait_row(reg, par))) break;
          next_row();
          const uint32_t rb = reg;
          if (two) {
            if (!(ok = wait_row(reg, par))) break;
            next_row();
          }
          const bool live = two && g.levels > 1 && g.W1 > 0;
          int64_t g0 = px0 * HW1 + (int64_t)j * g.W1 + out.skew[1];
          if (live) {
            CvAppend ap(row, tail1, ((int)(g0 & 7) + lane * HW1) & 7, g.W1);
            for (int pc = 0; pc < np; ++pc) {
              uint32_t va[16], vb[16], a[8], b[8], w[4];
              load(ra, pc, va);
              load(rb, pc, vb);
              tc::ld_wait();
              pack(va, i, pc, a);
              pack(vb, i + 1, pc, b);
#pragma unroll
              for (int k = 0; k < 4; ++k)
                w[k] = pack2<T>(pool4<T>(a[2 * k], b[2 * k]), pool4<T>(a[2 * k + 1], b[2 * k + 1]));
              uint4* up = reinterpret_cast<uint4*>(p1) + pc;
              if (j & 1) {                                        // with the row above: two words of level 2
                const uint4 t = *up;
                *reinterpret_cast<uint2*>(up) = make_uint2(pack2<T>(pool4<T>(t.x, w[0]), pool4<T>(t.y, w[1])),
                                                           pack2<T>(pool4<T>(t.z, w[2]), pool4<T>(t.w, w[3])));
              } else {
                *up = make_uint4(w[0], w[1], w[2], w[3]);
              }
              ap.put(w);
            }
            ap.end();
          }
          tc::fence_before();
          __syncwarp();
          free_row(ra);
          if (two) free_row(rb);
          if (!live) continue;
          tail1 = run_flush(sh1, out.lvl[1], g0, HW1, g.W1, (j - (i0 >> 1)) * g.W1, j == (i1 >> 1) - 1, rows, chunks, stg);
          if (!(j & 1) || g.levels < 3 || g.W2 == 0) continue;
          g0 = px0 * HW2 + (int64_t)j2 * g.W2 + out.skew[2];
          {
            CvAppend ap(row, tail2, ((int)(g0 & 7) + lane * HW2) & 7, g.W2);
            for (int pc = 0; pc < np; ++pc) {
              const uint2 t = *reinterpret_cast<const uint2*>(reinterpret_cast<const uint4*>(p1) + pc);
              const uint32_t w[2] = {t.x, t.y};
              uint2* up = reinterpret_cast<uint2*>(p2) + pc;
              if (j2 & 1) {                                       // with the row above: a word of level 3
                const uint2 o = *up;
                *reinterpret_cast<uint32_t*>(up) = pack2<T>(pool4<T>(o.x, w[0]), pool4<T>(o.y, w[1]));
              } else {
                *up = t;
              }
              ap.put(w);
            }
            ap.end();
          }
          tail2 = run_flush(sh2, out.lvl[2], g0, HW2, g.W2, (j2 - (i0 >> 2)) * g.W2, j2 == (i1 >> 2) - 1, rows, chunks, stg);
          if (!(j2 & 1) || g.levels < 4 || g.W3 == 0) continue;
          g0 = px0 * HW3 + (int64_t)j3 * g.W3 + out.skew[3];
          {
            CvAppend ap(row, tail3, ((int)(g0 & 7) + lane * HW3) & 7, g.W3);
            for (int pc = 0; pc < np; ++pc) {
              const uint32_t w[1] = {*reinterpret_cast<const uint32_t*>(reinterpret_cast<const uint2*>(p2) + pc)};
              ap.put(w);
            }
            ap.end();
          }
          tail3 = run_flush(sh3, out.lvl[3], g0, HW3, g.W3, (j3 - (i0 >> 3)) * g.W3, j3 == (i1 >> 3) - 1, rows, chunks, stg);
        }
      }
      if (!ok) break;
    }
  }
  if (*abort_flag && tid == 0) atomicOr(info, HS2_DEV_TIMEOUT);
  tc::fence_before();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCvTmemCols) : "memory");
  }
}

// ------------------------------------------------------------------- host ---
namespace {

int cv_check(int64_t E, int64_t K1, int64_t K2, int C, int H, int W, int dtype, int precision, int levels) {
  if (E < 0 || K1 < 0 || K2 < 0 || H <= 0 || W <= 0 || levels < 1 || levels > 4) {
    set_error("corr_volume: bad sizes E=%lld K1=%lld K2=%lld H=%d W=%d levels=%d", (long long)E, (long long)K1,
              (long long)K2, H, W, levels);
    return HS2_ERR_INVALID;
  }
  if (C != kCvC) {
    set_error("corr_volume: %d feature channels (the kernel contracts exactly 128)", C);
    return HS2_ERR_INVALID;
  }
  if (W > kCvMaxW) {
    set_error("corr_volume: W=%d exceeds %d (one image row per TMA box)", W, kCvMaxW);
    return HS2_ERR_INVALID;
  }
  if ((int64_t)H * W * kCvC >= (int64_t(1) << 31)) {
    set_error("corr_volume: H*W=%lld too large", (long long)H * W);
    return HS2_ERR_INVALID;
  }
  if (dtype != HS2_F16 && dtype != HS2_BF16) {
    set_error("corr_volume: fmaps must be float16 or bfloat16");
    return HS2_ERR_DTYPE;
  }
  if (precision != HS2_CV_NATIVE && precision != HS2_CV_E4M3) {
    set_error("corr_volume: unknown precision %d", precision);
    return HS2_ERR_INVALID;
  }
  return HS2_OK;
}

size_t cv_workspace(int64_t K1, int64_t K2, int H, int W, int precision) {
  const int64_t HW = (int64_t)H * W;
  const int es = precision == HS2_CV_E4M3 ? 1 : 2;
  size_t bytes = (size_t)(K1 + K2) * HW * kCvC * es;
  bytes = (bytes + 255) & ~size_t(255);
  if (precision == HS2_CV_E4M3) bytes += ((size_t)(K1 + K2) * HW * sizeof(float) + 255) & ~size_t(255);
  return bytes;
}

template <typename T, int P>
int cv_pack(const void* f, int64_t K, int HW, void* rows, float* scale, cudaStream_t s) {
  if (K == 0) return HS2_OK;
  dim3 grid((HW + 63) / 64, (unsigned)K);
  HS2_PROF("corr_pack", s);
  corr_pack_kernel<T, P><<<grid, 256, 0, s>>>(static_cast<const T*>(f), HW, rows, scale);
  HS2_LAUNCH_CHECK("corr_pack_kernel");
  return HS2_OK;
}

// Operand rows [K, HW, 128] as a 3-D tensor (channels innermost); a box is 128 bytes of
// channels x box_rows pixels of one frame, so rows past a frame's last pixel read as zero.
int cv_map(CUtensorMap* map, void* rows, int64_t K, int HW, int P, int box_rows) {
  const int esize = P == kE4M3 ? 1 : 2;
  const cuuint64_t dims[3] = {(cuuint64_t)kCvC, (cuuint64_t)HW, (cuuint64_t)K};
  const cuuint64_t strides[2] = {(cuuint64_t)kCvC * esize, (cuuint64_t)HW * kCvC * esize};
  const cuuint32_t box[3] = {(cuuint32_t)(128 / esize), (cuuint32_t)box_rows, 1};
  const CUtensorMapDataType t = P == kE4M3  ? CU_TENSOR_MAP_DATA_TYPE_UINT8
                                : P == kBF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                             : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  return tc::encode_tiled(map, t, 3, rows, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

template <int P, typename T>
int cv_launch(const CvGeom& g, void* rows1, void* rows2, const float* s1, const float* s2, int64_t K1, int64_t K2,
              const int64_t* ii, const int64_t* jj, CvOut out, int32_t* info, cudaStream_t s) {
  CUtensorMap amap, bmap;
  int rc;
  if ((rc = cv_map(&amap, rows1, K1, g.HW, P, 128))) return rc;
  if ((rc = cv_map(&bmap, rows2, K2, g.HW, P, g.RW))) return rc;
  const int64_t units = g.E * g.mtiles * g.splits;
  if (units == 0) return HS2_OK;
  static DeviceOnce once;
  int dev = 0;
  HS2_CUDA(cudaGetDevice(&dev));
  static std::atomic<int> sms[kMaxDevices];
  rc = once.run(dev, [&]() -> int {
    HS2_CUDA(cudaFuncSetAttribute(corr_volume_kernel<P, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  227 * 1024));
    int n = 0;
    HS2_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
    sms[dev].store(n);
    return HS2_OK;
  });
  if (rc) return rc;
  const int grid = (int)std::min<int64_t>(units, 2 * sms[dev].load());
  HS2_PROF("corr_volume", s);
  corr_volume_kernel<P, T><<<grid, kCvThreads, g.smem, s>>>(amap, bmap, ii, jj, K1, K2, s1, s2, g, out, info);
  HS2_LAUNCH_CHECK("corr_volume_kernel");
  return HS2_OK;
}

}  // namespace

}  // namespace hs2

extern "C" int hs2_corr_volume_workspace_size(int64_t k1, int64_t k2, int channels, int ht, int wd, int dtype,
                                              int precision, size_t* bytes) {
  using namespace hs2;
  if (!bytes) {
    set_error("corr_volume_workspace_size: null output");
    return HS2_ERR_INVALID;
  }
  const int rc = cv_check(0, k1, k2, channels, ht, wd, dtype, precision, 4);
  if (rc) return rc;
  *bytes = cv_workspace(k1, k2, ht, wd, precision);
  return HS2_OK;
}

extern "C" int hs2_corr_volume(const void* fmap1, int64_t k1, const void* fmap2, int64_t k2, int channels, int ht,
                               int wd, int dtype, const int64_t* ii, const int64_t* jj, int64_t num_pairs,
                               int precision, int levels, void* const* pyramid, int32_t* info, void* workspace,
                               size_t workspace_bytes, hs2_stream_t stream) {
  using namespace hs2;
  int rc = cv_check(num_pairs, k1, k2, channels, ht, wd, dtype, precision, levels);
  if (rc) return rc;
  if (num_pairs == 0) return HS2_OK;
  if (!fmap1 || !fmap2 || !ii || !jj || !pyramid || !info) {
    set_error("corr_volume: null pointer argument");
    return HS2_ERR_INVALID;
  }
  for (int l = 0; l < levels; ++l) {
    const int hl = ht >> l, wl = wd >> l;
    if (hl > 0 && wl > 0 && !pyramid[l]) {
      set_error("corr_volume: level %d output missing", l);
      return HS2_ERR_INVALID;
    }
  }
  const size_t need = cv_workspace(k1, k2, ht, wd, precision);
  if (!workspace || workspace_bytes < need) {
    set_error("corr_volume: workspace of %zu bytes required", need);
    return HS2_ERR_WORKSPACE;
  }
  if ((rc = bind_device(fmap1))) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  const int HW = ht * wd;
  const int es = precision == HS2_CV_E4M3 ? 1 : 2;
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  void* rows1 = ws;
  void* rows2 = ws + (size_t)k1 * HW * kCvC * es;
  float* sc1 = nullptr;
  float* sc2 = nullptr;
  if (precision == HS2_CV_E4M3) {
    size_t off = ((size_t)(k1 + k2) * HW * kCvC + 255) & ~size_t(255);
    sc1 = reinterpret_cast<float*>(ws + off);
    sc2 = sc1 + (size_t)k1 * HW;
  }
  CvOut out;
  for (int l = 0; l < 4; ++l) {
    const uintptr_t at = l < levels ? reinterpret_cast<uintptr_t>(pyramid[l]) : 0;
    out.lvl[l] = reinterpret_cast<uint16_t*>(at & ~(uintptr_t)15);
    out.skew[l] = (int)(at & 15) / 2;
  }
  const CvGeom g = cv_geom(ht, wd, num_pairs, levels, precision == HS2_CV_E4M3 ? 1 : 2);
  if (dtype == HS2_F16) {
    if (precision == HS2_CV_E4M3) {
      if ((rc = cv_pack<__half, kE4M3>(fmap1, k1, HW, rows1, sc1, s))) return rc;
      if ((rc = cv_pack<__half, kE4M3>(fmap2, k2, HW, rows2, sc2, s))) return rc;
      return cv_launch<kE4M3, __half>(g, rows1, rows2, sc1, sc2, k1, k2, ii, jj, out, info, s);
    }
    if ((rc = cv_pack<__half, kF16>(fmap1, k1, HW, rows1, nullptr, s))) return rc;
    if ((rc = cv_pack<__half, kF16>(fmap2, k2, HW, rows2, nullptr, s))) return rc;
    return cv_launch<kF16, __half>(g, rows1, rows2, nullptr, nullptr, k1, k2, ii, jj, out, info, s);
  }
  if (precision == HS2_CV_E4M3) {
    if ((rc = cv_pack<__nv_bfloat16, kE4M3>(fmap1, k1, HW, rows1, sc1, s))) return rc;
    if ((rc = cv_pack<__nv_bfloat16, kE4M3>(fmap2, k2, HW, rows2, sc2, s))) return rc;
    return cv_launch<kE4M3, __nv_bfloat16>(g, rows1, rows2, sc1, sc2, k1, k2, ii, jj, out, info, s);
  }
  if ((rc = cv_pack<__nv_bfloat16, kBF16>(fmap1, k1, HW, rows1, nullptr, s))) return rc;
  if ((rc = cv_pack<__nv_bfloat16, kBF16>(fmap2, k2, HW, rows2, nullptr, s))) return rc;
  return cv_launch<kBF16, __nv_bfloat16>(g, rows1, rows2, nullptr, nullptr, k1, k2, ii, jj, out, info, s);
}
