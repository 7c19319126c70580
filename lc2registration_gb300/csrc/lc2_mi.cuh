// lc2_mi.cuh -- normalised mutual information, the similarity of
// PatchSize 0 (src/Interpolator/interpolator.cu:617-622;
// src/cu_LC2/cu_lc2_3d.cu:868-923, 1196-1301):
//   NMI = (H(U) + H(M)) / H(U, M)
// over the virtual grid, with 256 bins per image between the image's own
// minimum and maximum, H(X) = -sum p ln p, p = count / voxels, and the joint
// histogram indexed ultrasound bin + 256 * high-resolution bin.
//
// One image is static (the fixed one resampled once): its bins and entropy
// are computed once per context, by kernels of their own. Per batch of transforms
// four kernels run: the range of the warped image (ordered-integer atomics, one
// pair per CTA), the joint histogram (all its bins in shared memory, added to
// the transform's 256 KB histogram at the end), the entropy sums of slices of
// each histogram (kMiParts CTAs per transform) and their combination in a
// fixed order. A range CTA owns a 32 x 8 tile over a chunk of slices, a
// histogram CTA takes 32 x 32 x 32 blocks in turn: the sampling bases of a
// chunk's or block's slices are computed up front, one per thread, so the slices
// then stream without barriers; the bases are those of the generic warp kernel
// (tile_base), so the warped values are bit-identical to it. Counts are exact
// integers and the double sums run in a fixed order, so the value does not
// depend on the launch shape or the batch.
#pragma once

#include "lc2_kernels.cuh"

namespace lc2 {

constexpr int kMiBins = 256;
constexpr int kMiHist = kMiBins * kMiBins;

struct MiParams {
  int mx, my, mz;         // warped (moving) image
  int vx, vy, vz;         // virtual grid
  int warped_is_high_res; // 1: key = static bin + 256 * warped bin; 0: the transpose
  int zchunk;             // slices per range CTA, <= kMiChunk
};

// Order-preserving float <-> unsigned maps for atomicMin / atomicMax.
__device__ __forceinline__ unsigned mi_ord(float f) {
  const unsigned u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float mi_unord(unsigned u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// Bin of v in [lo, hi]: round((v - lo) * (255 / (hi - lo))) with float
// operations rounded to nearest (cu_lc2_3d.cu:886-889, 913); all voxels go
// to bin 0 when hi == lo. The static image's bins take the same operations
// (k_mi_static_bins).
__host__ __device__ inline float mi_scale(float lo, float hi) {
  return hi > lo ? 255.0f / (hi - lo) : 0.0f;
}
__device__ __forceinline__ int mi_bin(float v, float lo, float s) {
  return (int)roundf(__fmul_rn(__fsub_rn(v, lo), s));
}

constexpr int kMiChunk = 64;  // most slices of a range CTA or histogram block
constexpr int kMiParts = 32;  // entropy CTAs per transform (8 warped bins each)

// Sampling base of slice zb + t (< ze) of a 32 x 8 tile, and where the slice
// samples (tile_where), in shared memory.
struct MiBases {
  int ib[kMiChunk][3];
  float fb[kMiChunk][3];
  float4 base[kMiChunk];
  int where[kMiChunk];
};
__device__ __forceinline__ void mi_base(const Xform* X, const MiParams& P, int x0, int y0, int zb,
                                        int ze, int t, MiBases& B) {
  if (zb + t < ze) {
    TileBase T;
    tile_base(X, x0, y0, zb + t, T);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      B.ib[t][a] = T.ib[a];
      B.fb[t][a] = T.fb[a];
    }
    B.base[t] = tile_inside_base(T, P.mx, P.my);
    B.where[t] = tile_where(T, P.mx, P.my, P.mz);
  }
}

template <typename TM, bool BIG>
__device__ __forceinline__ float mi_sample(const TM* __restrict__ mov, const MiParams& P,
                                           const float* A, const MiBases& B, int t, float dx,
                                           float dy) {
  const int where = B.where[t];
  if (where == kTileInside)
    return tile_sample_inside<TM, BIG>(mov, (unsigned)P.mx, (unsigned)P.mx * (unsigned)P.my, A,
                                       B.base[t], dx, dy);
  if (where == kTileOutside) return 0.0f;
  if (where == kTileEdge)
    return tile_sample_edge<TM>(mov, P.mx, P.my, P.mz, B.ib[t], A, B.fb[t], dx, dy);
  TileBase T;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    T.ib[a] = B.ib[t][a];
    T.fb[a] = B.fb[t][a];
  }
#pragma unroll
  for (int i = 0; i < 9; ++i) T.A[i] = A[i];
  return tile_sample<3, TM>(mov, P.mx, P.my, P.mz, T, (int)dx, (int)dy);
}

// Range of the static image: range[0] / [1] hold its ordered minimum / maximum
// (mi_ord), 0xffffffff and 0 before.
template <int = 0>
__global__ void __launch_bounds__(256) k_mi_static_range(const float* __restrict__ img, size_t n,
                                                         unsigned* __restrict__ range) {
  unsigned lo = 0xffffffffu, hi = 0;
  for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (size_t)gridDim.x * 256) {
    const unsigned u = mi_ord(img[i]);
    lo = min(lo, u);
    hi = max(hi, u);
  }
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  if ((threadIdx.x & 31) == 0) {
    atomicMin(range, lo);
    atomicMax(range + 1, hi);
  }
}

// Bins of the static image in that range, and how many voxels each holds.
template <int = 0>
__global__ void __launch_bounds__(256) k_mi_static_bins(const float* __restrict__ img, size_t n,
                                                        const unsigned* __restrict__ range,
                                                        unsigned char* __restrict__ bin,
                                                        unsigned long long* __restrict__ counts) {
  __shared__ unsigned s_n[kMiBins];
  s_n[threadIdx.x] = 0;  // 256 threads, 256 bins
  __syncthreads();
  const float lo = mi_unord(range[0]), sc = mi_scale(lo, mi_unord(range[1]));
  for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (size_t)gridDim.x * 256) {
    const int b = min(max(mi_bin(img[i], lo, sc), 0), kMiBins - 1);
    bin[i] = (unsigned char)b;
    atomicAdd(&s_n[b], 1u);
  }
  __syncthreads();
  if (s_n[threadIdx.x]) atomicAdd(counts + threadIdx.x, (unsigned long long)s_n[threadIdx.x]);
}

// Range of the warped image of each transform. Bound by the L1 lookups of its
// gathers, eight samples of a thread in flight as in k_presample (one at a time:
// 1028 us instead of 996 for the whole of 50 transforms at 128^3; eight instead
// of four in the histogram's loop: 14 us more). Grid (tiles of 32 x 8, z chunks,
// transforms), block (32, 8).
constexpr int kMiRangeAhead = 8;
template <typename TM, bool BIG>
__global__ void __launch_bounds__(256) k_mi_range(const TM* __restrict__ mov, MiParams P,
                                                  const Xform* __restrict__ xf, int k0,
                                                  unsigned* __restrict__ rmin,
                                                  unsigned* __restrict__ rmax) {
  __shared__ MiBases B;
  __shared__ float red[2][8];
  const int ntx = (P.vx + 31) / 32;
  const int x0 = (blockIdx.x % ntx) * 32, y0 = (blockIdx.x / ntx) * 8;
  const int zb = blockIdx.y * P.zchunk, ze = min(zb + P.zchunk, P.vz);
  const int slot = blockIdx.z;
  mi_base(xf + k0 + slot, P, x0, y0, zb, ze, threadIdx.y * 32 + threadIdx.x, B);
  float A[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) A[i] = __ldg(&xf[k0 + slot].ah[i]);
  __syncthreads();
  const int x = x0 + threadIdx.x, y = y0 + threadIdx.y;
  float lo = INFINITY, hi = -INFINITY;
  if (x < P.vx && y < P.vy) {
    const float dx = (float)threadIdx.x, dy = (float)threadIdx.y;
    int z = zb;
    for (; z + kMiRangeAhead <= ze; z += kMiRangeAhead) {
      float v[kMiRangeAhead];
#pragma unroll
      for (int k = 0; k < kMiRangeAhead; ++k) v[k] = mi_sample<TM, BIG>(mov, P, A, B, z + k - zb, dx, dy);
#pragma unroll
      for (int k = 0; k < kMiRangeAhead; ++k) {
        lo = fminf(lo, v[k]);
        hi = fmaxf(hi, v[k]);
      }
    }
    for (; z < ze; ++z) {
      const float v = mi_sample<TM, BIG>(mov, P, A, B, z - zb, dx, dy);
      lo = fminf(lo, v);
      hi = fmaxf(hi, v);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if (threadIdx.x == 0) {
    red[0][threadIdx.y] = lo;
    red[1][threadIdx.y] = hi;
  }
  __syncthreads();
  if (threadIdx.y == 0 && threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) {
      lo = fminf(lo, red[0][w]);
      hi = fmaxf(hi, red[1][w]);
    }
    if (hi >= lo) {
      atomicMin(rmin + k0 + slot, mi_ord(lo));
      atomicMax(rmax + k0 + slot, mi_ord(hi));
    }
  }
}

// Joint histogram of each transform: static bins sbin (uint8 per voxel) and
// the warped image's bins in its range. A CTA counts its share of a transform's
// 32 x 32 x kMiHistChunk blocks in shared memory, all 2^16 bins as 16-bit halves of
// 32-bit words (128 KB), and adds the non-zero ones to the global histogram at
// the end: with global atomics per voxel (merged per warp and, on large grids, in
// a shared table of 2048 keys) the histogram took twice the time of the same
// sampling without it. A half that reaches 2^15 is emptied into the global bin
// by the thread whose count crossed the mark; until it has, the CTA's other
// 1023 threads add at most what is left of the block, kMiHistChunk each, so a
// half never overflows. Grid (shares, transforms), 1024 threads.
constexpr int kMiHistThreads = 1024;
constexpr int kMiHistChunk = 32;
static_assert((kMiHistThreads - 1) * kMiHistChunk < (1 << 15) && kMiHistChunk <= kMiChunk, "");
constexpr size_t kMiHistBytes = sizeof(unsigned) * (kMiHist / 2);

template <typename TM, bool BIG>
__global__ void __launch_bounds__(kMiHistThreads, 1)
    k_mi_hist(const TM* __restrict__ mov, MiParams P, const Xform* __restrict__ xf, int k0,
              const unsigned char* __restrict__ sbin, const unsigned* __restrict__ rmin,
              const unsigned* __restrict__ rmax, unsigned* __restrict__ hist) {
  extern __shared__ unsigned s_hist[];
  __shared__ MiBases B[4];  // the block's four 32 x 8 tiles
  const int ntx = (P.vx + 31) / 32, nty = (P.vy + 31) / 32, nzc = (P.vz + kMiHistChunk - 1) / kMiHistChunk;
  const int slot = blockIdx.y, tid = threadIdx.x, lane = tid & 31, row = tid >> 5;
  const Xform* X = xf + k0 + slot;
  for (int i = tid; i < kMiHist / 2; i += kMiHistThreads) s_hist[i] = 0;
  float A[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) A[i] = __ldg(&X->ah[i]);
  const float lo = mi_unord(rmin[k0 + slot]), hi = mi_unord(rmax[k0 + slot]);
  const float sc = mi_scale(lo, hi);
  unsigned* h = hist + (size_t)(k0 + slot) * kMiHist;
  const MiBases& T = B[row >> 3];
  const float dx = (float)lane, dy = (float)(row & 7);
  auto count = [&](int wb, int sb) {
    if (wb < 0 || wb >= kMiBins) return;
    const int key = P.warped_is_high_res ? sb + kMiBins * wb : wb + kMiBins * sb;
    const int shift = 16 * (key & 1);
    const unsigned before = atomicAdd(&s_hist[key >> 1], 1u << shift) >> shift & 0xffffu;
    if (before == 0x7fffu) {
      atomicSub(&s_hist[key >> 1], 0x8000u << shift);
      atomicAdd(h + key, 0x8000u);
    }
  };
  for (long long blk = blockIdx.x; blk < (long long)ntx * nty * nzc; blk += gridDim.x) {
    const int zc = (int)(blk % nzc), t = (int)(blk / nzc);
    const int x0 = (t % ntx) * 32, y0 = (t / ntx) * 32, zb = zc * kMiHistChunk;
    const int ze = min(zb + kMiHistChunk, P.vz);
    __syncthreads();  // the previous block's bases are read
    if (tid < 4 * kMiHistChunk)
      mi_base(X, P, x0, y0 + 8 * (tid / kMiHistChunk), zb, ze, tid % kMiHistChunk,
              B[tid / kMiHistChunk]);
    __syncthreads();
    const int x = x0 + lane, y = y0 + row;
    if (x < P.vx && y < P.vy) {
      const unsigned char* sb = sbin + ((size_t)zb * P.vy + y) * P.vx + x;
      const size_t plane = (size_t)P.vx * P.vy;
      int z = zb;
      for (; z + 4 <= ze; z += 4) {
        float v[4];
        int b[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          v[k] = mi_sample<TM, BIG>(mov, P, A, T, z + k - zb, dx, dy);
          b[k] = sb[(size_t)(z + k - zb) * plane];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) count(mi_bin(v[k], lo, sc), b[k]);
      }
      for (; z < ze; ++z)
        count(mi_bin(mi_sample<TM, BIG>(mov, P, A, T, z - zb, dx, dy), lo, sc),
              sb[(size_t)(z - zb) * plane]);
    }
  }
  __syncthreads();
  for (int i = tid; i < kMiHist / 2; i += kMiHistThreads) {
    const unsigned w = s_hist[i];
    if (w & 0xffffu) atomicAdd(h + 2 * i, w & 0xffffu);
    if (w >> 16) atomicAdd(h + 2 * i + 1, w >> 16);
  }
}

// Entropy sums of one part of each joint histogram: part b holds the warped
// bins [8b, 8b + 8) -- the rows of the histogram (key = static + 256 warped)
// or its columns (key = warped + 256 static). part[k][b] = (sum over its
// joint bins of c ln c, sum over its warped marginals of c ln c). Grid
// (kMiParts, transforms), 256 threads.
// The histogram is left zeroed for the next batch.
__global__ void __launch_bounds__(256) k_mi_part(unsigned* __restrict__ hist, int k0,
                                                 int warped_is_high_res,
                                                 double* __restrict__ part) {
  constexpr int WB = kMiBins / kMiParts;  // warped bins per part
  __shared__ unsigned marg[WB];
  __shared__ double red[2][8];
  const int k = k0 + blockIdx.y, b = blockIdx.x, tid = threadIdx.x;
  unsigned* h = hist + (size_t)k * kMiHist;
  if (tid < WB) marg[tid] = 0;
  __syncthreads();
  double sj = 0.0;
#pragma unroll
  for (int j = 0; j < WB; ++j) {
    // rows: warped bin WB b + j, static bin tid; columns: warped bin
    // WB b + (tid & 7), static bin (tid >> 3) + 32 j
    const int wl = warped_is_high_res ? j : (tid & (WB - 1));
    const int sbn = warped_is_high_res ? tid : (tid >> 3) + 32 * j;
    const int w = WB * b + wl;
    unsigned* hc = warped_is_high_res ? h + (sbn + kMiBins * w) : h + (w + kMiBins * sbn);
    const unsigned c = *hc;
    if (c) {
      *hc = 0;
      sj += (double)c * log((double)c);
      atomicAdd(&marg[wl], c);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sj += __shfl_down_sync(0xffffffffu, sj, o);
  if ((tid & 31) == 0) red[0][tid >> 5] = sj;
  __syncthreads();
  if (tid == 0) {
    double a = 0.0, m = 0.0;
    for (int w = 0; w < 8; ++w) a += red[0][w];
    for (int i = 0; i < WB; ++i)
      if (marg[i]) m += (double)marg[i] * log((double)marg[i]);
    part[((size_t)k * kMiParts + b) * 2] = a;
    part[((size_t)k * kMiParts + b) * 2 + 1] = m;
  }
}

// NMI of each transform from its parts, summed in part order.
// h_static: entropy of the static image; voxels: virtual-grid size. The ranges
// are reset for the next batch; host_out and flag as in k_finalize.
__global__ void k_mi_nmi(const double* __restrict__ part, int cnt, double h_static,
                         double voxels, unsigned* __restrict__ rmin, unsigned* __restrict__ rmax,
                         double* __restrict__ out, double* __restrict__ host_out,
                         unsigned* __restrict__ flag) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < cnt) {
    double a = 0.0, b = 0.0;
    for (int i = 0; i < kMiParts; ++i) {
      a += part[((size_t)k * kMiParts + i) * 2];
      b += part[((size_t)k * kMiParts + i) * 2 + 1];
    }
    const double ln_n = log(voxels);
    const double hj = ln_n - a / voxels;  // H(U, M)
    const double hw = ln_n - b / voxels;  // H(warped)
    double v = (h_static + hw) / hj;
    if (isnan(v) || isinf(v)) v = 0.0;
    rmin[k] = 0xffffffffu;
    rmax[k] = 0u;
    out[k] = v;
    if (host_out) host_out[k] = v;
  }
  if (flag) raise_flag(flag);
}

}  // namespace lc2
