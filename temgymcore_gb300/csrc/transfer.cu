// transfer.cu - ray transfer through stacks of 5x5 matrices
// (transfer.py:6-112): every ray through the cumulative products of a matrix
// sequence, and a point source's fan through one matrix.
//
// The reference's helpers are float64 NumPy / JAX.  25 float64 multiply-adds
// per (ray, plane) against 40 written bytes would make the transfer float64-
// pipe bound on GB300 (float64 issues at ~1/64 of the float32 rate), so the
// stack transfer runs in double-float arithmetic: every matrix entry and ray
// component as an unevaluated float32 pair (hi + lo, 48 significant bits),
// products with their exact rounding error (FMA), sums with TwoSum, and the
// result rounded back to float64 with integer operations.  Errors stay at a
// few 2^-47 of the sum of the term magnitudes; a ray or matrix with a nonzero
// entry outside [2^-39, 2^62] (where a product's error term would leave the
// normal float32 range) takes the float64 path.
#include <cstring>

#include "tg_common.cuh"

namespace tg {

constexpr int kMaxTransfer = 120;  // matrices per call (24 KB of kernel parameters)

// Zero pattern of a cumulative product: TR_FULL (none assumed), TR_AFFINE (last
// row 0 0 0 0 c), TR_SPLIT (besides, x and y do not mix: rows x, dx use columns x,
// dx, 1 and rows y, dy columns y, dy, 1; a column without a rotated element).  A
// zero entry's product and sum are exact no-ops on a finite ray, so leaving them
// out changes no result.
enum TrClass : uint8_t { TR_FULL = 0, TR_AFFINE = 1, TR_SPLIT = 2 };

struct TransferMats {
  int32_t m;
  int32_t pad;
  double c[kMaxTransfer][25];  // cumulative products, row-major
  uint8_t cls[kMaxTransfer];   // TrClass of each
};

// ---------------------------------------------------------------- double-float
struct DF {
  float h, l;
};

// a float64 value inside the double-float range (zero, or |v| in [2^-39, 2^62])
__host__ __device__ inline bool df_range(double v) {
  const double a = v < 0 ? -v : v;
  return v == 0.0 || (a >= 1.8189894035458565e-12 && a <= 4.611686018427388e18);
}

// a * b: the product of the heads with its exact rounding error, plus the
// cross terms (lo * lo is below the precision kept)
__device__ __forceinline__ DF df_mul(DF a, DF b) {
  const float p = __fmul_rn(a.h, b.h);
  float e = __fmaf_rn(a.h, b.h, -p);
  e = __fmaf_rn(a.h, b.l, e);
  e = __fmaf_rn(a.l, b.h, e);
  return DF{p, e};
}

// a + b: TwoSum of the heads, the tails added to the error; the pair is
// left unrenormalised (a short sum of products stays within a few 2^-47 of
// the term magnitudes) and df_norm is applied once per result
__device__ __forceinline__ DF df_add(DF a, DF b) {
  const float s = __fadd_rn(a.h, b.h);
  const float bb = __fsub_rn(s, a.h);
  const float err = __fadd_rn(__fsub_rn(a.h, __fsub_rn(s, bb)), __fsub_rn(b.h, bb));
  return DF{s, __fadd_rn(err, __fadd_rn(a.l, b.l))};
}

// Fast2Sum renormalisation: |lo| <= ulp(hi) / 2 afterwards
__device__ __forceinline__ DF df_norm(DF a) {
  const float h = __fadd_rn(a.h, a.l);
  return DF{h, __fsub_rn(a.l, __fsub_rn(h, a.h))};
}

// hi + lo rounded to the nearest float64 (far below the pair's own 2^-47; cut off
// instead, the mean error is 0.31 ulp against 0.17), without float64 operations.  For a renormalised pair
// |lo| <= ulp32(hi) / 2, so in units of hi's float64 ulp, 2^(e - 52), lo is a
// number below 2^28: lo times the power of two, rounded to an integer, is added to
// hi's float64 bits.  A lo that reduces a power of two leaves hi's binade, where
// the grid is twice as fine and lo counts double.  |hi| < 2^-74 (no such power of
// two in float32; zero) and non-finite parts take the general rounding.
__device__ __forceinline__ double df_to_double(float h, float l) {
  const uint32_t hb = __float_as_uint(h), lb = __float_as_uint(l);
  if ((hb & 0x7fffffffu) - (53u << 23) >= (202u << 23)) {
    if ((hb << 1) == 0u) return __longlong_as_double((long long)((uint64_t)(hb + lb) << 32));  // lo is 0 too
    return add_f64_f32(f32_to_f64(h), l);
  }
  uint32_t scale = 0x99000000u - (hb & 0xff800000u);  // 2^(52 - e) with hi's sign
  if ((hb & 0x7fffffu) == 0u && (int32_t)(hb ^ lb) < 0) scale += 1u << 23;
  const int n = __float2int_rn(__fmul_rn(l, __uint_as_float(scale)));
  // hi's float64 bits: exponent rebiased (+ 896 << 20), significand widened
  const uint32_t dhi = (uint32_t)((((int32_t)hb >> 3) & (int32_t)0x8fffffff) + 0x38000000), dlo = hb << 29;
  return __longlong_as_double((long long)(((uint64_t)dhi << 32) | dlo) + (long long)n);
}

// ------------------------------------------------- two double-floats at a time
// (packed pairs: the component of x and the component of y)
// A pair of ray components, with the negated parts that the products below use.
struct Ray2 {
  F2 h, nh, nl;
};
__device__ __forceinline__ Ray2 ray2(DF a, DF b) {
  return Ray2{f2(a.h, b.h), f2(-a.h, -b.h), f2(-a.l, -b.l)};
}
// A pair of double-floats as (hi, -lo): the error of a product then needs no
// negation, h v - p = -(p + h (-v)).
struct DF2 {
  F2 h, nl;
};
__device__ __forceinline__ DF2 df2_mul(const ulonglong2& c, const Ray2& v) {  // c = (hi, hi), (lo, lo)
  const F2 ch{c.x}, cl{c.y};
  const F2 p = f2_mul(ch, v.h);
  return DF2{p, f2_fma(cl, v.nh, f2_fma(ch, v.nl, f2_fma(ch, v.nh, p)))};
}
__device__ __forceinline__ DF2 df2_add(DF2 a, DF2 b) {  // df_add
  const F2 s = f2_add(a.h, b.h), bb = f2_sub(s, a.h);
  const F2 err = f2_add(f2_sub(a.h, f2_sub(s, bb)), f2_sub(b.h, bb));
  return DF2{s, f2_sub(f2_add(a.nl, b.nl), err)};
}

// The split of a float64 inside the double-float range, with integer operations:
// the head is the value rounded to 24 bits (ties away from zero), the tail the
// signed rest in units of 2^(e - 52), rounded to 24 bits.  False for a value
// outside the range (2^62 itself too), whose split means nothing.
__device__ __forceinline__ bool df_component(double v, DF& out) {
  const uint64_t b = (uint64_t)__double_as_longlong(v);
  const uint32_t hi = (uint32_t)(b >> 32), lo = (uint32_t)b, e = (hi >> 20) & 0x7ffu, sign = hi & 0x80000000u;
  const uint32_t top = ((hi & 0x7fffffffu) << 3 | lo >> 29) - (896u << 23);  // exponent and 23 bits
  const int rest = (int)(lo << 3) >> 3;                                       // the low 29 bits, signed
  const bool zero = ((hi << 1) | lo) == 0u;
  out.h = zero ? 0.0f : __uint_as_float(sign | (top + ((lo >> 28) & 1u)));
  out.l = zero ? 0.0f : __fmul_rn(__int2float_rn(rest), __uint_as_float(sign | ((e - 948u) << 23)));
  return zero || e - (1023u - 39u) < 101u;
}

constexpr int kTrThreads = 256;
constexpr int kTrMinBlocks = 4;
constexpr int kTrWaves = 4;       // blocks per SM and wave aimed at
constexpr int kTrPlanes = 4;      // planes between two writes
constexpr int kTrStride = 22;     // doubles per ray in a warp's buffer: 4 records of 5, 16-byte aligned
constexpr int kTrWarpDoubles = 32 * kTrStride;
constexpr int kTrVec = 5 * kTrPlanes / 2;    // 16-byte vectors of a ray's records
constexpr int kTrWriteRays = 32 / kTrVec;    // whole rays in a warp's write
static_assert(kTrPlanes % 2 == 0 && kTrStride % 2 == 0 && kTrStride >= 5 * kTrPlanes && kTrWriteRays >= 1, "");
constexpr int kTrTab = 13;        // 16-byte entries of a plane's split matrix

// out[n][p][i] = sum_j C[p][i][j] ray[n][j] in double-float.  A thread keeps one
// ray's split components in registers and walks planes [p0, p1) of its block
// row, so that a warp reads each matrix entry once (a broadcast) and skips a
// plane's zero entries together.  The rows of x and y (and of dx and dy) are a
// packed pair: row x takes columns x, y, dx, dy, 1 and row y columns y, x, dy,
// dx, 1.  Four planes' records of the warp's rays are collected in shared memory
// and leave as 16-byte vectors, 160 contiguous bytes a ray.  Bound by the
// instructions issued (8 a term and pair, 20 to round a result).  Measured at
// 1 M rays x 16 planes (6 planes split, 10 affine): 208 us; 399 with one
// (ray, plane) pair per thread, 25 terms each, and a float64 conversion run for
// every result ahead of its branch (52 % of the float64 pipe).
__global__ void __launch_bounds__(kTrThreads, kTrMinBlocks)
k_transfer_rays_df(const __grid_constant__ TransferMats T, int64_t n, int planes_per_block,
                   const double* __restrict__ rays, double* __restrict__ out, int vec) {
  extern __shared__ __align__(16) double trm[];  // [warps][32][kTrStride] records, then the planes' split matrices
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int p0 = blockIdx.y * planes_per_block, p1 = min(T.m, p0 + planes_per_block);
  double* rec = trm + warp * kTrWarpDoubles;
  ulonglong2* mc = reinterpret_cast<ulonglong2*>(trm + kTrThreads / 32 * kTrWarpDoubles);
  // entries 0..4: rows x and y, 5..9: rows dx and dy, 10..12: the last row's five
  for (int i = threadIdx.x; i < (p1 - p0) * kTrTab; i += kTrThreads) {
    const int p = i / kTrTab, e = i - p * kTrTab;
    const double* c = T.c[p0 + p];
    double a, b;
    if (e < 10) {
      const int row = e < 5 ? 0 : 2, j = e < 5 ? e : e - 5;
      a = c[row * 5 + j];
      b = c[row * 5 + 5 + (j == 4 ? 4 : j ^ 1)];
    } else {
      const int j = (e - 10) * 2;
      a = c[20 + j];
      b = j < 4 ? c[21 + j] : 0.0;
    }
    DF da, db;  // in range: the host's rule
    df_component(a, da);
    df_component(b, db);
    mc[i] = make_ulonglong2(f2(da.h, db.h).u, f2(da.l, db.l).u);
  }
  __syncthreads();
  const int sub = lane / kTrVec, off = lane - sub * kTrVec;  // a write takes the records of kTrWriteRays rays
  const int64_t stride = (int64_t)gridDim.x * kTrThreads;
  for (int64_t r0 = (int64_t)blockIdx.x * kTrThreads + warp * 32; r0 < n; r0 += stride) {  // the warp's 32 rays
    const int64_t r = r0 + lane;
    const double* src = rays + 5 * (r < n ? r : n - 1);
    DF v[5];
    bool ok = true;
#pragma unroll
    for (int j = 0; j < 5; ++j) ok &= df_component(__ldg(src + j), v[j]);
    const Ray2 xy = ray2(v[0], v[1]), yx = ray2(v[1], v[0]), sxy = ray2(v[2], v[3]), syx = ray2(v[3], v[2]),
               one = ray2(v[4], v[4]);
    const int live = (int)(n - r0 < 32 ? n - r0 : 32);
    for (int pc = p0; pc < p1; pc += kTrPlanes) {
      const int np = min(kTrPlanes, p1 - pc);
      for (int q = 0; q < np; ++q) {
        const ulonglong2* c = mc + (pc - p0 + q) * kTrTab;
        double* o = rec + lane * kTrStride + 5 * q;
        const int cls = T.cls[pc + q];  // the same for the whole block
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          DF2 a = df2_mul(c[5 * i], xy);
          if (cls == TR_SPLIT) {
            a = df2_add(a, df2_mul(c[5 * i + 2], sxy));
          } else {
            a = df2_add(a, df2_mul(c[5 * i + 1], yx));
            a = df2_add(a, df2_mul(c[5 * i + 2], sxy));
            a = df2_add(a, df2_mul(c[5 * i + 3], syx));
          }
          a = df2_add(a, df2_mul(c[5 * i + 4], one));
          const F2 h = f2_sub(a.h, a.nl);  // df_norm
          const F2 nl = f2_add(a.nl, f2_sub(h, a.h));
          o[2 * i] = df_to_double(f2_lo(h), -f2_lo(nl));
          o[2 * i + 1] = df_to_double(f2_hi(h), -f2_hi(nl));
        }
        const float* cf = reinterpret_cast<const float*>(c + 10);  // h, h, l, l of two entries
        DF acc = df_mul(DF{cf[8], cf[10]}, v[4]);
        if (cls == TR_FULL) {
          DF sum = df_mul(DF{cf[0], cf[2]}, v[0]);
#pragma unroll
          for (int j = 1; j < 4; ++j)
            sum = df_add(sum, df_mul(DF{cf[(j >> 1) * 4 + (j & 1)], cf[(j >> 1) * 4 + 2 + (j & 1)]}, v[j]));
          acc = df_add(sum, acc);
        }
        acc = df_norm(acc);
        o[4] = df_to_double(acc.h, acc.l);
        if (!ok) {  // outside the double-float range: float64
          const double* c64 = T.c[pc + q];
#pragma unroll 1
          for (int i = 0; i < 5; ++i)
            o[i] = c64[5 * i + 0] * src[0] + c64[5 * i + 1] * src[1] + c64[5 * i + 2] * src[2] +
                   c64[5 * i + 3] * src[3] + c64[5 * i + 4] * src[4];
        }
      }
      __syncwarp();
      const int64_t pitch = (int64_t)T.m * 5;
      double* dst = out + r0 * pitch + pc * 5;
      if (vec && np == kTrPlanes) {  // m and pc even, out 16-byte aligned
        const double* from = rec + sub * kTrStride + 2 * off;
        double* to = dst + sub * pitch + 2 * off;
        for (int ray = sub; ray < live && sub < kTrWriteRays;
             ray += kTrWriteRays, from += kTrWriteRays * kTrStride, to += kTrWriteRays * pitch)
          *reinterpret_cast<double2*>(to) = *reinterpret_cast<const double2*>(from);
      } else {
        const int per = 5 * np;  // doubles of a ray
        for (int i = lane; i < live * per; i += 32) {
          const int ray = i / per, k = i - ray * per;
          dst[(int64_t)ray * pitch + k] = rec[ray * kTrStride + k];
        }
      }
      __syncwarp();
    }
  }
}

// out[n][p][i] = sum_j C[p][i][j] ray[n][j], one (ray, plane) pair per thread:
// a warp writes 32 consecutive 40-byte records.
__global__ void __launch_bounds__(256)
k_transfer_rays(const __grid_constant__ TransferMats T, int64_t n, const double* __restrict__ rays,
                double* __restrict__ out) {
  __shared__ double sc[kMaxTransfer * 25];
  for (int i = threadIdx.x; i < T.m * 25; i += blockDim.x) sc[i] = T.c[i / 25][i % 25];
  __syncthreads();
  const int64_t total = n * (int64_t)T.m;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = t / T.m;
    const int p = (int)(t - r * T.m);
    const double* v = rays + r * 5;
    const double v0 = v[0], v1 = v[1], v2 = v[2], v3 = v[3], v4 = v[4];
    const double* c = sc + p * 25;
    double* o = out + t * 5;
#pragma unroll
    for (int i = 0; i < 5; ++i)
      o[i] = c[5 * i + 0] * v0 + c[5 * i + 1] * v1 + c[5 * i + 2] * v2 + c[5 * i + 3] * v3 +
             c[5 * i + 4] * v4;
  }
}

struct PtSrcArgs {
  double x0, y0;
  double t[25];
  int64_t n;
  const double *sx, *sy;
  double* out;  // [4][n]
};

// rows x, y, dx, dy of T [x0, y0, sx, sy, 1] for every slope pair
__global__ void __launch_bounds__(256) k_transfer_pt_src(const __grid_constant__ PtSrcArgs A) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < A.n;
       k += (int64_t)gridDim.x * blockDim.x) {
    const double v[5] = {A.x0, A.y0, A.sx[k], A.sy[k], 1.0};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      double s = 0.0;
#pragma unroll
      for (int j = 0; j < 5; ++j) s += A.t[5 * i + j] * v[j];
      A.out[(int64_t)i * A.n + k] = s;
    }
  }
}

static int sm_count_transfer() {
  static int cached = 0;
  if (!cached) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&cached, cudaDevAttrMultiProcessorCount, dev);
    if (cached <= 0) cached = 148;
  }
  return cached;
}

static void mat5(const double* a, const double* b, double* out) {
  double t[25];
  for (int i = 0; i < 5; ++i)
    for (int j = 0; j < 5; ++j) {
      double s = 0.0;
      for (int k = 0; k < 5; ++k) s += a[5 * i + k] * b[5 * k + j];
      t[5 * i + j] = s;
    }
  std::memcpy(out, t, sizeof(t));
}

}  // namespace tg

using namespace tg;

extern "C" int tg_transfer_cumulative(int32_t m, const double* matrices, double* cumulative) {
  if (m <= 0 || !matrices || !cumulative) return TG_ERR_INVALID;
  // transfer.py:150-183: start from the LAST matrix and multiply the earlier
  // ones on the left: cumulative[k] = M[m-1-k] @ ... @ M[m-1]
  double total[25];
  std::memcpy(total, matrices + (int64_t)(m - 1) * 25, sizeof(total));
  std::memcpy(cumulative, total, sizeof(total));
  for (int k = 1; k < m; ++k) {
    mat5(matrices + (int64_t)(m - 1 - k) * 25, total, total);
    std::memcpy(cumulative + (int64_t)k * 25, total, sizeof(total));
  }
  return TG_OK;
}

extern "C" int tg_transfer_rays(int64_t n, const double* rays, int32_t m, const double* matrices,
                                double* out, void* stream) {
  if (n < 0 || m <= 0 || !matrices) return TG_ERR_INVALID;
  if (m > kMaxTransfer) return TG_ERR_TOO_LARGE;
  if (n > 0 && (!rays || !out)) return TG_ERR_INVALID;
  TransferMats T;
  std::memset(&T, 0, sizeof(T));
  T.m = m;
  int st = tg_transfer_cumulative(m, matrices, &T.c[0][0]);
  if (st != TG_OK) return st;
  if (n == 0) return TG_OK;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  bool df = true;
  for (int i = 0; i < m * 25 && df; ++i) df = df_range((&T.c[0][0])[i]);
  if (df) {
    for (int p = 0; p < m; ++p) {
      const double* c = T.c[p];
      auto zero = [&](int i, int j) { return c[5 * i + j] == 0.0; };
      bool affine = true, split = true;
      for (int j = 0; j < 4; ++j) affine = affine && zero(4, j);
      for (int i = 0; i < 4; ++i) split = split && zero(i, 1 - (i & 1)) && zero(i, 3 - (i & 1));
      T.cls[p] = affine ? (split ? TR_SPLIT : TR_AFFINE) : TR_FULL;
    }
    // all planes a thread where the rays fill the GPU, else fewer (a multiple
    // of kTrPlanes) over more blocks
    const int64_t rblocks = (n + kTrThreads - 1) / kTrThreads, want = (int64_t)sm_count_transfer() * 4 * kTrWaves;
    int64_t rows = (want + rblocks - 1) / rblocks;
    const int groups = (m + kTrPlanes - 1) / kTrPlanes;
    if (rows > groups) rows = groups;
    int per = (int)((groups + rows - 1) / rows) * kTrPlanes;
    // Few rays: one plane a thread while a single wave holds every block, two up
    // to half a wave.  us, one or two planes / four: 1 ray x 7 planes 2.9 / 5.0,
    // 1,000 x 3 3.5 / 6.0, 1,000 x 61 4.3 / 7.4, 5,000 x 5 3.7 / 7.2, 20,000 x 7 6.2 / 8.2;
    // 30,000 x 8 and 20,000 x 12 (472 of 608 blocks) as two 9.0 / 8.0.
    const int64_t wave = (int64_t)sm_count_transfer() * kTrMinBlocks;
    if (rblocks * m <= wave) per = 1;
    else if (rblocks * ((m + 1) / 2) <= wave / 2) per = 2;
    const size_t smem = sizeof(double) * (kTrThreads / 32) * kTrWarpDoubles +
                        sizeof(ulonglong2) * kTrTab * (size_t)(per < m ? per : m);  // at most 70 KB
    const int smem_max = (int)(sizeof(double) * (kTrThreads / 32) * kTrWarpDoubles + sizeof(ulonglong2) * kTrTab * kMaxTransfer);
    if (smem_opt_in<k_transfer_rays_df>(smem_max) != cudaSuccess) return TG_ERR_CUDA;
    const int vec = (m & 1) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
    const dim3 grid((unsigned)(rblocks < want ? rblocks : want), (unsigned)((m + per - 1) / per));
    k_transfer_rays_df<<<grid, kTrThreads, smem, s>>>(T, n, per, rays, out, vec);
    return cudaGetLastError() == cudaSuccess ? TG_OK : TG_ERR_CUDA;
  }
  const int64_t total = n * (int64_t)m;
  int64_t blocks = (total + 255) / 256;
  const int64_t cap = (int64_t)sm_count_transfer() * 8;
  if (blocks > cap) blocks = cap;
  k_transfer_rays<<<(int)blocks, 256, 0, s>>>(T, n, rays, out);
  return cudaGetLastError() == cudaSuccess ? TG_OK : TG_ERR_CUDA;
}

extern "C" int tg_transfer_rays_pt_src(double x0, double y0, int64_t n, const double* slopes_x,
                                       const double* slopes_y, const double* matrix, double* out,
                                       void* stream) {
  if (n < 0 || !matrix) return TG_ERR_INVALID;
  if (n > 0 && (!slopes_x || !slopes_y || !out)) return TG_ERR_INVALID;
  if (n == 0) return TG_OK;
  PtSrcArgs A;
  A.x0 = x0;
  A.y0 = y0;
  std::memcpy(A.t, matrix, sizeof(A.t));
  A.n = n;
  A.sx = slopes_x;
  A.sy = slopes_y;
  A.out = out;
  int64_t blocks = (n + 255) / 256;
  const int64_t cap = (int64_t)sm_count_transfer() * 8;
  if (blocks > cap) blocks = cap;
  k_transfer_pt_src<<<(int)blocks, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(A);
  return cudaGetLastError() == cudaSuccess ? TG_OK : TG_ERR_CUDA;
}
