// scan.cu - 4D-STEM batch: one ray bundle traced through the model at every
// scan position (probe), binned into one dense detector image per probe.
//
// This replaces the reference's per-scan-position Python loop of
// run_to_end (run.py:85-116) + Detector.into_image (grid.py:231-280).
//
// Kernel layout: a persistent grid walks the probes; one CTA owns one probe
// at a time.  The CTA
//   1. derives the probe's scan position (float64, from the ScanGrid pixel
//      map or an explicit list) and the per-probe Scanner/Descanner shifts,
//   2. traces the bundle (L2-resident, read by every CTA) in registers and
//      keeps each ray's packed pixel in shared memory,
//   3. reduces the hits' bounding box and histograms it in a shared-memory
//      window, in bands of as many box rows as fit the window (one band in
//      the usual case: a probe lights a small disc; wider ones where that pays,
//      ScanArgs::bands),
//   4. writes the dense image once: the window rows, and a quarter of the
//      image's rows of zeros around them, as 16-byte stores; the other rows
//      are all zeros and leave as TMA bulk copies from a zero buffer in
//      shared memory (asynchronous: the CTA goes on to the next probe while
//      the copy engine streams them).  Both write paths run at once.
// Small images and large bundles run k_scan_image instead (scan_use_image): the
// probe's whole image as packed 16-bit counters in shared memory, written out
// once.  What takes neither (wide discs on a large image, more than 65,535 rays)
// is zero-filled and counted with global atomics.  The HBM
// traffic is therefore the dense histogram write, ~h*w*4 bytes/probe.
#include <cstring>

#include "tg_common.cuh"

TG_DEFINE_ERROR_WORD(scan)

namespace tg {

constexpr int kScanThreads = 256;
constexpr int kMaxSmemRays = 4096;  // packed pixels kept in shared memory
constexpr int kZeroBytes = 8192;    // zero source of the bulk row copies
constexpr int kSmallBox = 5632;     // bins of a box that always takes the window (one band)
// k_scan_hist's shared memory (four CTAs fill an SM): the zero source, the
// packed pixels, and the rest as the window's 16-bit counters (16,000 bins
// beside 4,096 rays, 22,000 beside 1,024)
constexpr int kHistSmem = 56 * 1024 - 512;

struct ScanArgs {
  int64_t n;  // rays per probe
  const float *x, *y, *dx, *dy;
  double z_scalar;
  int32_t n_probes, cols;
  double t[6];
  const double* positions;
  int32_t* hist;  // [n_probes][h][w]
  float* probe_xy;  // optional [n_probes][2][n]
  int32_t h, w;
  int32_t vec4;  // rows are 16-byte aligned: dense write with int4 stores
  int32_t vec_in;  // the bundle's arrays (and probe_xy's rows) are 16-byte aligned: four consecutive rays a thread
  int32_t bulk;  // images in device memory: zero rows as TMA bulk copies
  int32_t win_bins;    // k_scan_hist's window (16-bit counters)
  int32_t bands;       // boxes above kSmallBox bins take the window up to this many twentieths of the rows
  int32_t store_rows;  // zero rows next to the window written by stores, not bulk copies
};

__device__ __forceinline__ void probe_shifts(const Program& P, const ScanArgs& A, int p,
                                             float4* pshift) {
  double spx, spy;
  if (A.positions) {
    spx = A.positions[2 * (size_t)p];
    spy = A.positions[2 * (size_t)p + 1];
  } else {
    double r = (double)(p / A.cols), c = (double)(p % A.cols);
    spy = __dadd_rn(__dadd_rn(__dmul_rn(A.t[0], r), __dmul_rn(A.t[1], c)), A.t[2]);
    spx = __dadd_rn(__dadd_rn(__dmul_rn(A.t[3], r), __dmul_rn(A.t[4], c)), A.t[5]);
  }
  for (int k = 0; k < P.n_probe_ops; ++k) {
    const double* q = P.pcoef[k];
    pshift[k] = make_float4((float)(q[0] * spx + q[1] * spy + q[2]),
                            (float)(q[3] * spx + q[4] * spy + q[5]),
                            (float)(q[6] * spx + q[7] * spy + q[8]),
                            (float)(q[9] * spx + q[10] * spy + q[11]));
  }
}

// The rays of one thread's turn: R consecutive rays from R * t (read as one
// vector per array) with A.vec_in, else rays t, t + threads, ... of the
// block's R * threads.
template <int R, typename I>
__device__ __forceinline__ I scan_ray(const ScanArgs& A, I base, int k) {
  return A.vec_in ? base + R * (int)threadIdx.x + k : base + (int)threadIdx.x + k * (int)blockDim.x;
}

// R rays of the turn at base through the probe's chain to pixels: hit[k] says
// whether ray k counts (alive, inside the detector).  Those at or past n are
// traced from zeros and never hit.  I: the index type (32 bits where the host
// bounds n).
template <int R, typename I>
__device__ __forceinline__ void trace_rays(const Program& P, const ScanArgs& A, const BinCoef& B,
                                           const float4* pshift, int p, I base, bool write_xy,
                                           int (&py)[R], int (&px)[R], bool (&hit)[R]) {
  static_assert(R == 4, "one 16-byte vector per array");
  const I n = (I)A.n, i0 = scan_ray<R>(A, base, 0);
  const int step = A.vec_in ? 1 : (int)blockDim.x;
  RayS r[R];
  float dv[R];  // the bundle starts from one plane: no per-ray first distance
  uint64_t sb[R];
  bool alive[R];
  const bool vec = A.vec_in && i0 + R - 1 < n;
  if (vec) {
    const float4 x = __ldg(reinterpret_cast<const float4*>(A.x + i0)), y = __ldg(reinterpret_cast<const float4*>(A.y + i0));
    const float4 u = __ldg(reinterpret_cast<const float4*>(A.dx + i0)), v = __ldg(reinterpret_cast<const float4*>(A.dy + i0));
    r[0] = RayS{x.x, y.x, u.x, v.x, 0.f};
    r[1] = RayS{x.y, y.y, u.y, v.y, 0.f};
    r[2] = RayS{x.z, y.z, u.z, v.z, 0.f};
    r[3] = RayS{x.w, y.w, u.w, v.w, 0.f};
  } else {
#pragma unroll
    for (int k = 0; k < R; ++k) {
      const I i = i0 + k * step;
      const bool in = i < n;
      r[k] = RayS{in ? A.x[i] : 0.f, in ? A.y[i] : 0.f, in ? A.dx[i] : 0.f, in ? A.dy[i] : 0.f, 0.f};
    }
  }
#pragma unroll
  for (int k = 0; k < R; ++k) {
    dv[k] = 0.f;
    sb[k] = 0;
    alive[k] = true;
  }
  chain_forward_n<R>(P, pshift, r, dv, sb, alive, &P.aber[0][0]);
  if (write_xy) {
    float* ox = A.probe_xy + (size_t)p * 2 * A.n;
    if (vec) {
      *reinterpret_cast<float4*>(ox + i0) = make_float4(r[0].x, r[1].x, r[2].x, r[3].x);
      *reinterpret_cast<float4*>(ox + A.n + i0) = make_float4(r[0].y, r[1].y, r[2].y, r[3].y);
    } else {
#pragma unroll
      for (int k = 0; k < R; ++k) {
        const I i = i0 + k * step;
        if (i < n) {
          ox[i] = r[k].x;
          ox[A.n + i] = r[k].y;
        }
      }
    }
  }
  float x[R], y[R];
  bool live[R], nonfinite[R];
#pragma unroll
  for (int k = 0; k < R; ++k) {
    x[k] = r[k].x;
    y[k] = r[k].y;
    live[k] = i0 + k * step < n;
  }
  bin_rays<R>(x, y, B, live, py, px, nonfinite);
#pragma unroll
  for (int k = 0; k < R; ++k) {
    const bool in = live[k];
    hit[k] = in && alive[k] && (unsigned)py[k] < (unsigned)A.h && (unsigned)px[k] < (unsigned)A.w;
    if (in && nonfinite[k]) atomicOr(&g_tg_err, TG_EW_NONFINITE);
  }
}

constexpr int kScanRays = 4;  // rays a thread traces together

// Bounding box of the hits over the CTA (rows mn[0] .. mx[0], columns mn[1]
// .. mx[1]; mx[0] < 0: no hit): one barrier for all four bounds.
__device__ __forceinline__ void block_box(int& rmin, int& rmax, int& cmin, int& cmax, int4* red) {
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  const int4 v = make_int4(__reduce_min_sync(0xffffffffu, rmin), __reduce_max_sync(0xffffffffu, rmax),
                           __reduce_min_sync(0xffffffffu, cmin), __reduce_max_sync(0xffffffffu, cmax));
  if (l == 0) red[w] = v;
  __syncthreads();
  int4 t = red[0];
  for (int i = 1; i < (int)(blockDim.x >> 5); ++i) {
    const int4 o = red[i];
    t = make_int4(min(t.x, o.x), max(t.y, o.y), min(t.z, o.z), max(t.w, o.w));
  }
  rmin = t.x; rmax = t.y; cmin = t.z; cmax = t.w;
}

__global__ void __launch_bounds__(kScanThreads, 4)
k_scan_hist(const __grid_constant__ Program P, const __grid_constant__ ScanArgs A,
            const __grid_constant__ BinCoef B) {
  // zero source | packed pixels (py << 16) | px, or 0xffffffff = no hit | window
  extern __shared__ __align__(128) uint32_t smem[];
  __shared__ float4 pshift[kMaxProbeOps];
  __shared__ int4 red[kScanThreads / 32];
  const int64_t n = A.n;
  const bool fits = n <= kMaxSmemRays;
  const int H = A.h, W = A.w;
  uint32_t* pix = smem + kZeroBytes / 4;
  uint32_t* win = pix + (fits ? ((int)n + 3) / 4 * 4 : 0);  // 16-bit counters in pairs
  for (int i = threadIdx.x; i < kZeroBytes / 4; i += blockDim.x) smem[i] = 0u;
  // the bulk copies read the zero source through the async proxy
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();
  const uint32_t zsrc = smem_u32(smem);
  // one CTA per probe (two row bands per probe as separate work items
  // measured 0.186 vs 0.179 ms on the 64x64-probe workload: the doubled trace
  // and barriers cost more than the finer balance gains)
  for (int p = blockIdx.x; p < A.n_probes; p += gridDim.x) {
    if (threadIdx.x == 0) probe_shifts(P, A, p, pshift);
    __syncthreads();
    int rmin = 0x7fffffff, rmax = -1, cmin = 0x7fffffff, cmax = -1;
    for (int64_t i = 0; i < n; i += kScanThreads * kScanRays) {
      int py[kScanRays], px[kScanRays];
      bool ok[kScanRays];
      trace_rays<kScanRays>(P, A, B, pshift, p, i, A.probe_xy != nullptr, py, px, ok);
#pragma unroll
      for (int k = 0; k < kScanRays; ++k) {
        const int64_t j = scan_ray<kScanRays>(A, i, k);
        if (fits && j < n) pix[j] = ok[k] ? ((uint32_t)py[k] << 16) | (uint32_t)px[k] : 0xffffffffu;
        if (ok[k]) {
          rmin = min(rmin, py[k]); rmax = max(rmax, py[k]);
          cmin = min(cmin, px[k]); cmax = max(cmax, px[k]);
        }
      }
    }
    block_box(rmin, rmax, cmin, cmax, red);
    int32_t* img = A.hist + (size_t)p * H * W;
    const bool any = rmax >= 0;
    // window columns [c0, c0 + wc): whole groups of four pixels, so that a
    // group's counters are one aligned pair of words
    const int c0 = any ? cmin & ~3 : 0, wc = any ? ((cmax - c0) | 3) + 1 : 0;
    const int rows_hit = any ? rmax - rmin + 1 : 0, cols_hit = any ? cmax - cmin + 1 : 0;
    const bool small = (int64_t)rows_hit * cols_hit <= kSmallBox;
    if (fits && wc <= A.win_bins && (small || rows_hit * 20 <= H * A.bands)) {
      // rows [r0, r1) are written by stores: the box rows and, with bulk
      // copies, store_rows zero rows around them; the rows outside are zeros:
      // bulk copies of the zero buffer (row starts are 16-byte aligned: W is a
      // multiple of 4 and the images 16-byte aligned); one thread issues them,
      // the group is committed and left in flight.  Images in host memory
      // (written across the host link) take stores for every row instead.
      int r0 = A.bulk ? (any ? rmin : 0) : 0, r1 = A.bulk ? (any ? rmax + 1 : 0) : H;
      if (A.bulk && A.store_rows > 0) {  // store_rows more zero rows by stores, around the window
        int below = min(A.store_rows >> 1, r0);
        const int above = min(A.store_rows - below, H - r1);
        below = min(A.store_rows - above, r0);
        r0 -= below;
        r1 += above;
      }
      if (A.bulk && threadIdx.x == 0) {
        char* base = reinterpret_cast<char*>(img);
        const int64_t row_bytes = (int64_t)W * 4;
        const int64_t spans[2][2] = {{0, r0 * row_bytes}, {r1 * row_bytes, H * row_bytes}};
        for (int sp = 0; sp < 2; ++sp)
          for (int64_t off = spans[sp][0]; off < spans[sp][1]; off += kZeroBytes) {
            const int64_t left = spans[sp][1] - off;
            const uint32_t bytes = (uint32_t)(left < kZeroBytes ? left : kZeroBytes);
            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                         :: "l"(base + off), "r"(zsrc), "r"(bytes) : "memory");
          }
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        // keep at most four items' copies in flight (a hardware wait on
        // the copy engine, no polling)
        asm volatile("cp.async.bulk.wait_group.read 4;" ::: "memory");
      }
      // the box in bands of as many rows as the window holds (a disc wider
      // than the window re-reads its packed pixels once per band)
      const int band_rows = any ? A.win_bins / wc : H;
      int lo = r0;  // first row not yet written
      int b0 = any ? rmin : 0;
      do {
        const int b1 = any ? min(b0 + band_rows, rmax + 1) : 0;  // box rows [b0, b1) of this band
        const int hi = any && b1 <= rmax ? b1 : r1;              // the last band writes the trailing zero rows
        if (any) {
          for (int i = threadIdx.x; i < ((b1 - b0) * wc) >> 1; i += blockDim.x) win[i] = 0u;
          __syncthreads();
          for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const uint32_t v = pix[i];
            const int py = (int)(v >> 16), px = (int)(v & 0xffffu);
            if (v != 0xffffffffu && py >= b0 && py < b1) {
              const int bin = (py - b0) * wc + (px - c0);
              atomicAdd(&win[bin >> 1], (bin & 1) ? 0x10000u : 1u);
            }
          }
          __syncthreads();
        }
        if (A.vec4) {
          // window rows: counts inside the window's columns, zeros elsewhere
          const int w4 = W >> 2;
          const int total = (hi - lo) * w4;
          int4* rows = reinterpret_cast<int4*>(img) + (int64_t)lo * w4;
          for (int i = threadIdx.x; i < total; i += blockDim.x) {
            const int row = lo + i / w4, c = ((i % w4) << 2) - c0;
            int4 v = make_int4(0, 0, 0, 0);
            if (row >= b0 && row < b1 && c >= 0 && c < wc) {
              const uint2 t = *reinterpret_cast<const uint2*>(win + (((row - b0) * wc + c) >> 1));
              v = make_int4((int)(t.x & 0xffffu), (int)(t.x >> 16), (int)(t.y & 0xffffu), (int)(t.y >> 16));
            }
            __stcs(rows + i, v);
          }
        } else {
          // A thread's row and column advance by the block's width in rows and
          // columns.  (One division by W a pixel: 301 x 301 images, 625 probes of 64
          // rays, 90 us in 32 bits, 127 in 64.)  h, w <= 65,535: fewer than 2^32 -
          // 2^16 pixels.
          const uint32_t total = (uint32_t)(hi - lo) * (uint32_t)W;
          const int dr = kScanThreads / W, dc = kScanThreads - dr * W;
          int row = lo + (int)threadIdx.x / W, c = (int)threadIdx.x % W - c0;
          int32_t* px = img + (int64_t)lo * W;
          for (uint32_t i = threadIdx.x; i < total; i += kScanThreads) {
            int v = 0;
            if (row >= b0 && row < b1 && c >= 0 && c < wc) {
              const int bin = (row - b0) * wc + c;
              v = (int)((win[bin >> 1] >> (16 * (bin & 1))) & 0xffffu);
            }
            __stcs(px + i, v);
            row += dr;
            c += dc;
            if (c >= W - c0) {
              c -= W;
              ++row;
            }
          }
        }
        lo = hi;
        b0 = b1;
        if (any && b0 <= rmax) __syncthreads();  // the window is reused by the next band
      } while (any && b0 <= rmax);
    } else {
      // slow path: zero the image, then global atomics (re-trace if needed)
      const int64_t total = (int64_t)H * W, odd = (int64_t)(-(reinterpret_cast<uintptr_t>(img) >> 2) & 3);
      const int64_t head = odd < total ? odd : total, vecs = (total - head) >> 2;  // 16-byte stores from img + head on
      int4* body = reinterpret_cast<int4*>(img + head);
      for (int64_t i = threadIdx.x; i < vecs; i += kScanThreads) body[i] = make_int4(0, 0, 0, 0);
      if (threadIdx.x < head) img[threadIdx.x] = 0;
      if (threadIdx.x < total - head - 4 * vecs) img[head + 4 * vecs + threadIdx.x] = 0;
      __syncthreads();
      if (fits) {
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
          const uint32_t v = pix[i];
          if (v != 0xffffffffu) atomicAdd(img + (int64_t)(v >> 16) * W + (int)(v & 0xffffu), 1);
        }
      } else {
        for (int64_t i = 0; i < n; i += kScanThreads * kScanRays) {
          int py[kScanRays], px[kScanRays];
          bool ok[kScanRays];
          trace_rays<kScanRays>(P, A, B, pshift, p, i, false, py, px, ok);
#pragma unroll
          for (int k = 0; k < kScanRays; ++k)
            if (ok[k]) atomicAdd(img + (int64_t)py[k] * W + px[k], 1);
        }
      }
    }
    __syncthreads();  // shared buffers are reused by the next item
  }
  // every bulk copy has read the zero source and written its rows before the CTA exits
  if (A.bulk && threadIdx.x == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// One CTA per probe with the whole image as 16-bit counters packed in pairs
// (h * w * 2 bytes of shared memory; a probe's rays are at most 65,535, so no
// counter overflows): the rays are traced once, each hit is one shared
// atomic, and the image leaves as 16-byte stores that also clear the counters
// for the next probe.  Any disc costs the same.  Bound by the issue of the
// trace for many rays a probe and by the image write for few (400 MB of images:
// 69 us, 0.86 of measured HBM).  40 x 36 probes x 10,000 rays, an 80-pixel disc
// on 192 x 192: 392 us with a zero fill and global atomics, 77 here.
template <int T, int kPerSm>
__global__ void __launch_bounds__(T, kPerSm)
k_scan_image(const __grid_constant__ Program P, const __grid_constant__ ScanArgs A,
             const __grid_constant__ BinCoef B) {
  extern __shared__ __align__(16) uint32_t cnt[];  // [(h * w + 1) / 2], padded to a multiple of 2 words
  __shared__ float4 pshift[kMaxProbeOps];
  const int bins = A.h * A.w, W = A.w, words = ((bins + 3) >> 2) << 1;
  for (int i = threadIdx.x; i < words; i += T) cnt[i] = 0u;
  for (int p = blockIdx.x; p < A.n_probes; p += gridDim.x) {
    if (threadIdx.x == 0) probe_shifts(P, A, p, pshift);
    __syncthreads();  // the shifts; the counters cleared by the previous probe's write
    for (int i = 0; i < A.n; i += T * kScanRays) {
      int py[kScanRays], px[kScanRays];
      bool ok[kScanRays];
      trace_rays<kScanRays>(P, A, B, pshift, p, i, A.probe_xy != nullptr, py, px, ok);
#pragma unroll
      for (int k = 0; k < kScanRays; ++k)
        if (ok[k]) {
          const int b = py[k] * W + px[k];
          atomicAdd(cnt + (b >> 1), (b & 1) ? 0x10000u : 1u);
        }
    }
    __syncthreads();
    int32_t* img = A.hist + (size_t)p * bins;
    if (A.vec4) {
      uint2* c2 = reinterpret_cast<uint2*>(cnt);
      for (int i = threadIdx.x; i < (bins >> 2); i += T) {
        const uint2 v = c2[i];
        c2[i] = make_uint2(0u, 0u);
        __stcs(reinterpret_cast<int4*>(img) + i,
               make_int4((int)(v.x & 0xffffu), (int)(v.x >> 16), (int)(v.y & 0xffffu), (int)(v.y >> 16)));
      }
    } else {  // two pixels a thread: consecutive lanes write consecutive pairs
      for (int i = threadIdx.x; i < (bins + 1) >> 1; i += T) {
        const uint32_t v = cnt[i];
        cnt[i] = 0u;
        __stcs(img + 2 * i, (int)(v & 0xffffu));
        if (2 * i + 1 < bins) __stcs(img + 2 * i + 1, (int)(v >> 16));
      }
    }
    // the next probe's shifts are written before its first barrier, which
    // every thread reaches only after its part of this write
  }
}

static int sm_count_scan() {
  static int cached = 0;
  if (!cached) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&cached, cudaDevAttrMultiProcessorCount, dev);
    if (cached <= 0) cached = 148;
  }
  return cached;
}

// k_scan_image's counters with six, three and two CTAs an SM
constexpr size_t kImageSmem6 = 36 * 1024, kImageSmem3 = 75 * 1024, kImageSmem2 = 112 * 1024;

// Dynamic shared memory one CTA may opt into beside k_scan_image's static
// per-probe shifts.
static size_t scan_smem_max() {
  static size_t cached = 0;
  if (!cached) {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cached = (size_t)(v > 49152 ? v : 49152) - kMaxProbeOps * sizeof(float4);
  }
  return cached;
}

// Whole-image counters (k_scan_image) or the window (k_scan_hist)?  Measured
// on 400 MB of images, us, window / whole image, for a disc of 9 pixels and
// one of 0.42 of the detector:
//   128 x 128, 512 rays: 83 / 69 and 113 / 69;   4,096 rays: 182 / 113 and 213 / 112
//   192 x 192, 1,024:    68 / 74 and 90 / 69;    2,048: 68 / 69 and 107 / 69;  4,096: 93 / 85 and 141 / 85
//   256 x 256, 1,024:    68 / 129 and 80 / 107;  4,096: 72 / 92 and 114 / 92
// A counter array that leaves room for six CTAs an SM always wins, one that
// leaves room for three wins or ties from 2,048 rays on; larger ones hold too
// few warps while the window has room for the packed pixels.  (A call without
// rays takes the window: there is nothing to count.)
static bool scan_use_image(int64_t n, size_t smem) {
  if (n <= 0 || n > 65535 || smem > scan_smem_max()) return false;
  return n > kMaxSmemRays || smem <= kImageSmem6 || (smem <= kImageSmem3 && n >= 2048);
}

template <int T, int kPerSm>
static int scan_image_launch(const Program& P, const ScanArgs& A, const BinCoef& B, size_t smem, cudaStream_t s) {
  if (smem_opt_in<k_scan_image<T, kPerSm>>((int)scan_smem_max()) != cudaSuccess) return TG_ERR_CUDA;
  const int res = sm_count_scan() * kPerSm;
  k_scan_image<T, kPerSm><<<res < A.n_probes ? res : A.n_probes, T, smem, s>>>(P, A, B);
  return cudaGetLastError() == cudaSuccess ? TG_OK : TG_ERR_CUDA;
}

}  // namespace tg

using namespace tg;

extern "C" int tg_scan_hist(const tg_model* model, const tg_rays* bundle, const tg_scan* scan,
                            const tg_grid* grid, int32_t* hist, float* probe_xy, void* stream) {
  if (!model || !bundle || !scan || !grid) return TG_ERR_INVALID;
  if (!hist && scan->n_probes > 0) return TG_ERR_INVALID;
  if (bundle->n < 0 || scan->n_probes < 0 || grid->h <= 0 || grid->w <= 0) return TG_ERR_INVALID;
  if (grid->h > 65535 || grid->w > 65535) return TG_ERR_TOO_LARGE;
  if (!scan->positions && scan->cols <= 0) return TG_ERR_INVALID;
  if (bundle->z) return TG_ERR_UNSUPPORTED;  // one source plane for the bundle
  if (bundle->n > 0 && (!bundle->x || !bundle->y || !bundle->dx || !bundle->dy))
    return TG_ERR_INVALID;
  Program P;
  int st = compile_program(model, false, bundle->z_scalar, &P);
  if (st != TG_OK) return st;
  if (scan->n_probes == 0) return TG_OK;
  ScanArgs A;
  std::memset(&A, 0, sizeof(A));
  A.n = bundle->n;
  A.x = bundle->x; A.y = bundle->y; A.dx = bundle->dx; A.dy = bundle->dy;
  A.z_scalar = bundle->z_scalar;
  A.n_probes = scan->n_probes;
  A.cols = scan->cols;
  for (int i = 0; i < 6; ++i) A.t[i] = scan->t[i];
  A.positions = scan->positions;
  A.hist = hist;
  A.probe_xy = probe_xy;
  A.h = grid->h;
  A.w = grid->w;
  A.vec4 = ((grid->w & 3) == 0) && ((reinterpret_cast<uintptr_t>(hist) & 15) == 0);
  auto a16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  A.vec_in = a16(A.x) && a16(A.y) && a16(A.dx) && a16(A.dy) && (!probe_xy || (a16(probe_xy) && (A.n & 3) == 0));
  // a quarter of the rows go out as stores beside the bulk copies: the two
  // write paths run in parallel (256x256 images, 64x64 probes: 0.1815 ms with
  // bulk copies alone, 0.1777 ms with 64 stored rows; 32 and 80 rows between)
  A.store_rows = grid->h / 4;
  bool on_host = false;
  {  // images may live in pinned host memory (written by the kernel across the host link)
    cudaPointerAttributes pa;
    if (cudaPointerGetAttributes(&pa, hist) != cudaSuccess) return TG_ERR_CUDA;
    on_host = pa.type == cudaMemoryTypeHost;
    A.bulk = A.vec4 && pa.type == cudaMemoryTypeDevice;
    if (pa.type != cudaMemoryTypeDevice && pa.type != cudaMemoryTypeHost && pa.type != cudaMemoryTypeManaged)
      return TG_ERR_INVALID;  // unregistered host memory
  }
  BinCoef B = make_bincoef(grid);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const size_t img_smem = ((size_t)grid->h * grid->w + 3) / 4 * 8;
  if (scan_use_image(A.n, img_smem)) {
    A.vec4 = (((int64_t)grid->h * grid->w) & 3) == 0 && ((reinterpret_cast<uintptr_t>(hist) & 15) == 0);
    // as many CTAs an SM as their counters allow, the fewer the larger
    if (img_smem <= kImageSmem6) return scan_image_launch<256, 6>(P, A, B, img_smem, s);
    if (img_smem <= kImageSmem3) return scan_image_launch<512, 3>(P, A, B, img_smem, s);
    if (img_smem <= kImageSmem2) return scan_image_launch<768, 2>(P, A, B, img_smem, s);
    return scan_image_launch<1024, 1>(P, A, B, img_smem, s);
  }
  A.win_bins = (kHistSmem - kZeroBytes - (A.n <= kMaxSmemRays ? (int)(A.n + 3) / 4 * 16 : 0)) / 4 * 2;
  if (smem_opt_in<k_scan_hist>(kHistSmem) != cudaSuccess) return TG_ERR_CUDA;
  static int per_sm = 0;  // residency, queried once
  if (!per_sm) {
    int q = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&q, k_scan_hist, kScanThreads, kHistSmem);
    per_sm = q > 0 ? q : 1;
  }
  int blocks = sm_count_scan() * per_sm;
  // Larger boxes: a zero fill with a global atomic a hit, or the window in bands?
  // The window leaves the zero rows to the bulk copies, which pays when every SM
  // holds its four CTAs and enough rows are left to them.  The bands' time over the
  // other's, 1,024 to 4,096 rays a probe:
  //   200 x 200, 625-12,321 probes: 100 rows 0.85-1.05, 130 rows 1.0-1.2
  //   256 x 256, 625-7,569:  130 rows 0.82-1.07, 160 rows 0.84-1.17, all rows 0.99-1.4
  //   300 x 300, 625-5,476:  160 rows 0.76-0.93, 200 rows 0.79-1.0, all rows 0.95-1.13
  //   512 x 512, 625-1,849:  300 rows 0.72-0.93, 400 rows 0.84-1.01, all rows 0.95-1.11
  // with one CTA an SM (81 probes, 512 x 512) 1.1 for 100 rows, 1.9 for all, and for
  // images of 160 x 160, which stay in L2, 1.1 to 1.6.  Rows of odd widths have no
  // bulk copies (301 x 301, 625 probes: 1.3-1.6).  Images in host memory take the bands always:
  // an atomic there crosses the host link.
  const int64_t pixels = (int64_t)grid->h * grid->w;
  if (on_host)
    A.bands = 20;
  else if (!A.bulk || scan->n_probes < blocks || pixels < 200 * 200)
    A.bands = 0;
  else
    A.bands = pixels < 300 * 300 ? 12 : 15;
  if (blocks > scan->n_probes) blocks = scan->n_probes;
  k_scan_hist<<<blocks, kScanThreads, kHistSmem, s>>>(P, A, B);
  return cudaGetLastError() == cudaSuccess ? TG_OK : TG_ERR_CUDA;
}
