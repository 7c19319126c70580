// lc2_quad2d.cuh -- 2D windows (2D and 2D-to-3D) in column quads.
#pragma once

#include "lc2_quad.cuh"

namespace lc2 {

// k_fused_quad's quads, planes and passes for one slice: a CTA resamples its
// 32 x TY tile's region, then a thread per halo quad (four rows of a column)
// forms the Sobel magnitudes and limbs of its points, the x window pass runs in
// place on pairs of rows, and the solving threads sum the y windows of four
// rows each. Same samples, integers and solve as fused_tile_2d, so the same
// bits.
template <int TY, int R, int NL = kLimbs>
struct Quad2D {
  static constexpr int R_ = R, W = 2 * R + 1;
  static constexpr int HX = 32 + 2 * R, HY = TY + 2 * R;
  static constexpr int NQ = (HY + 3) / 4;                     // halo quads per column
  static constexpr int TAIL = 2 * R * NQ;                     // quads of the columns beyond 32
  static constexpr int NT = 32 * (NQ + (TAIL + 31) / 32);
  static constexpr int PW = HX + 2, PH = HY + 2;              // resampled region
  // plane pitch = 2 or 6 mod 8: the tail warps' quads (rows 4 apart) read
  // distinct banks
  static constexpr int SP = PW + (6 - PW % 4) % 4;
  static constexpr int SR = 4 * NQ + 2;
  static constexpr int YP = 4 * (NQ | 1);                     // limb planes [column][row]
  // plane stride: consecutive (limb, pair) jobs of the x pass on consecutive banks
  static constexpr int PY = HX * YP + (64 + 4 * NQ - HX * YP % 32) % 32;
  static constexpr int XJOBS = NL * 2 * NQ;                   // x pass: (limb, pair of rows)
  static constexpr int ST = 32 * (TY / kQuadOut);             // solving threads
  static constexpr int NV = (kQuadOut + W - 1 + 3) / 4;       // quads a solving thread reads
  static constexpr size_t OFF_A = ((sizeof(float) * SP * SR + 15) / 16) * 16;
  static constexpr size_t BYTES = OFF_A + sizeof(int) * (size_t)NL * PY;
  static constexpr int CTAS = NT <= 256 ? 3 : 2;              // CTAs per SM compiled for
  static_assert(SP >= PW && SP % 4 == 2 && PY % 4 == 0 && PY >= HX * YP, "");
  static_assert(ST <= NT && TY / 4 - kQuadOut / 4 + NV <= NQ, "a solve stays in the plane");
};

// x window pass in place over the limb planes: two rows of one limb per job.
template <typename G>
__device__ __forceinline__ void quad2d_xpass(int* __restrict__ A) {
#pragma unroll 1
  for (int job = threadIdx.x; job < G::XJOBS; job += G::NT) {
    const int L = job / (2 * G::NQ);
    int* a = A + (size_t)L * G::PY + 2 * (job - L * (2 * G::NQ));
    int2 v[G::HX];
    int2 w = make_int2(0, 0);
#pragma unroll
    for (int i = 0; i < G::HX; ++i) {
      v[i] = *reinterpret_cast<const int2*>(a + i * G::YP);
      if (i < G::W) {
        w.x += v[i].x;
        w.y += v[i].y;
      } else {
        w.x += v[i].x - v[i - G::W].x;
        w.y += v[i].y - v[i - G::W].y;
      }
      if (i >= G::W - 1) *reinterpret_cast<int2*>(a + (i - G::W + 1) * G::YP) = w;
    }
  }
}

// Centred sums of kQuadOut outputs (quad_centred for 2D patches).
template <typename G>
__device__ __forceinline__ void quad2d_centred(const int* __restrict__ y, int L, const int* a,
                                               const int* b, long long* d) {
  using C = PatchConst<2, G::R_>;
  constexpr int n = (int)C::N, nk = (int)(C::N << C::K);
  int lo[kQuadOut], hi[kQuadOut];
  quad_window<G>(y + (size_t)L * G::PY, lo);
  quad_window<G>(y + (size_t)(L + 1) * G::PY, hi);
#pragma unroll
  for (int j = 0; j < kQuadOut; ++j)
    d[j] = (long long)hi[j] * nk + (long long)lo[j] * n - (long long)a[j] * b[j];
}

// Column and quad of a moments thread; whether it has one.
template <typename G>
__device__ __forceinline__ bool quad2d_of(int tid, int& hx, int& q) {
  if (tid < 32 * G::NQ) {
    hx = tid & 31;
    q = tid >> 5;
    return true;
  }
  const int t = tid - 32 * G::NQ;
  q = t / (2 * G::R_);
  hx = 32 + t - q * (2 * G::R_);
  return t < G::TAIL;
}

// One 32 x TY output tile of a 2D window; returns this thread's fixed-point
// measure sum. Ends with the shared planes still in use.
template <int WND, typename TM, typename TS, int TY, int R>
__device__ __forceinline__ long long quad_tile_2d(const TM* __restrict__ mov,
                                                  const TS* __restrict__ Ust,
                                                  const float* __restrict__ sig,
                                                  const int* __restrict__ su,
                                                  const FusedParams& P, const Xform* X, int tile,
                                                  unsigned char* smem_raw, TileShared& T,
                                                  float* __restrict__ out_measure) {
  using G = Quad2D<TY, R>;
  constexpr int KB = PatchConst<2, R>::K;
  constexpr unsigned kmask = (1u << KB) - 1u;
  float* mc = reinterpret_cast<float*>(smem_raw);
  int* A = reinterpret_cast<int*>(smem_raw + G::OFF_A);
  const int tid = threadIdx.x;
  const int x0 = (tile % P.ntx) * 32, y0 = (tile / P.ntx) * TY;
  const int gx0 = x0 - R - 1, gy0 = y0 - R - 1;
  // sampling base (x0 - R - 1, 32 floor(y0 / 32) - R - 1), as fused_tile_2d
  const int yb = y0 & 31;
  if (tid == 0) {
#pragma unroll
    for (int i = 0; i < 9; ++i) T.A[i] = X->ah[i];
    T.inside =
        region_base<WND, G::PW, G::PH>(*X, T.A, P, gx0, gy0, yb, 0, true, T.ib, T.fb) ? 1 : 0;
  }
  int hx, q;
  const bool own = quad2d_of<G>(tid, hx, q);
  // the quad's ultrasound, in flight while the tile is resampled
  float u[4];
  {
    const int gx = x0 - R + hx, gy = y0 - R + 4 * q;
    const bool xin = own && gx >= 0 && gx < P.vx;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      u[i] = (xin && gy + i >= 0 && gy + i < P.vy) ? ldf(Ust, (size_t)(gy + i) * P.vx + gx) : 0.0f;
  }
  __syncthreads();
  if (T.inside) {
    // all of a thread's samples in flight before the first is stored (5 % of
    // the kernel)
    constexpr int K = (G::PW * G::PH + G::NT - 1) / G::NT;
    float v[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int i = min(tid + k * G::NT, G::PW * G::PH - 1);
      const int py = i / G::PW, px = i - py * G::PW;
      if constexpr (WND == 3)
        v[k] = fused_sample_inside<TM>(mov, P, T.A, T.ib, T.fb, px, py + yb);
      else
        v[k] = fused_sample_inside2<TM>(mov, P, T.A, T.ib, T.fb, px, py + yb);
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int i = min(tid + k * G::NT, G::PW * G::PH - 1);
      const int py = i / G::PW, px = i - py * G::PW;
      mc[py * G::SP + px] = v[k];
    }
  } else {
    for (int i = tid; i < G::PW * G::PH; i += G::NT) {
      const int py = i / G::PW, px = i - py * G::PW;
      const int gx = gx0 + px, gy = gy0 + py;
      float v = 0.0f;
      if (gx >= 0 && gx < P.vx && gy >= 0 && gy < P.vy)
        v = fused_sample<WND, TM>(mov, P, T.A, T.ib, T.fb, px, py + yb);
      mc[py * G::SP + px] = v;
    }
  }
  __syncthreads();
  if (own) {
    const float* c = mc + (4 * q + 1) * G::SP + hx + 1;
    float l[6], m[6], r[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) {
      l[j] = c[(j - 1) * G::SP - 1];
      m[j] = c[(j - 1) * G::SP];
      r[j] = c[(j - 1) * G::SP + 1];
    }
    int qu[4], qm[4], qg[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {  // fused_sobel<2>
      const float gx = (r[i] - l[i]) + 2.0f * (r[i + 1] - l[i + 1]) + (r[i + 2] - l[i + 2]);
      const float gy = (l[i + 2] - l[i]) + 2.0f * (m[i + 2] - m[i]) + (r[i + 2] - r[i]);
      qg[i] = quant(sqrt_approx(gx * gx + gy * gy), P.qg);
      qm[i] = quant(m[i + 1], P.qm);
      qu[i] = quant(u[i], P.qu);
    }
    int* a = A + hx * G::YP + 4 * q;
    *reinterpret_cast<int4*>(a) = make_int4(qm[0], qm[1], qm[2], qm[3]);
    *reinterpret_cast<int4*>(a + G::PY) = make_int4(qg[0], qg[1], qg[2], qg[3]);
    auto put = [&](int k, const int* x, const int* y) {
      long long p[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) p[i] = (long long)x[i] * y[i];
      *reinterpret_cast<int4*>(a + k * G::PY) =
          make_int4((int)((unsigned)p[0] & kmask), (int)((unsigned)p[1] & kmask),
                    (int)((unsigned)p[2] & kmask), (int)((unsigned)p[3] & kmask));
      *reinterpret_cast<int4*>(a + (k + 1) * G::PY) = make_int4(
          (int)(p[0] >> KB), (int)(p[1] >> KB), (int)(p[2] >> KB), (int)(p[3] >> KB));
    };
    put(2, qu, qm);
    put(4, qu, qg);
    put(6, qm, qm);
    put(8, qg, qg);
    put(10, qm, qg);
  }
  // this thread's outputs: rows row0 .. row0 + 3 of column lane
  const int lane = tid & 31, row0 = kQuadOut * (tid >> 5);
  const int x = x0 + lane, yr = y0 + row0;
  const int rows = (tid < G::ST && x < P.vx) ? min(kQuadOut, P.vy - yr) : 0;
  float sg[kQuadOut];
  int sv[kQuadOut];
  float top = 0.0f;
#pragma unroll
  for (int j = 0; j < kQuadOut; ++j) {
    sg[j] = 0.0f;
    sv[j] = 0;
    if (j < rows) {
      sg[j] = __ldg(sig + (size_t)(yr + j) * P.vx + x);
      sv[j] = __ldg(su + (size_t)(yr + j) * P.vx + x);
    }
  }
  __syncthreads();
  quad2d_xpass<G>(A);
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kQuadOut; ++j) top = fmaxf(top, sg[j]);
  float ms[kQuadOut];
#pragma unroll
  for (int j = 0; j < kQuadOut; ++j) ms[j] = 0.0f;
  long long acc_m = 0;
  if (__any_sync(0xffffffffu, top > 0.0f)) {
    const int* yv = A + (size_t)lane * G::YP + row0;
    int aM[kQuadOut], aG[kQuadOut];
    float im[kQuadOut], ig[kQuadOut], rmg[kQuadOut], rum[kQuadOut];
    unsigned km = 0, kg = 0;
    long long d[kQuadOut];
    quad_window<G>(yv, aM);
    quad_window<G>(yv + G::PY, aG);
    quad2d_centred<G>(yv, 6, aM, aM, d);
#pragma unroll
    for (int j = 0; j < kQuadOut; ++j) {
      if (d[j] > P.thr_m) km |= 1u << j;
      im[j] = rsqrt_ftz(ll2f(d[j]));
    }
    quad2d_centred<G>(yv, 8, aG, aG, d);
#pragma unroll
    for (int j = 0; j < kQuadOut; ++j) {
      if (d[j] > P.thr_g) kg |= 1u << j;
      ig[j] = rsqrt_ftz(ll2f(d[j]));
    }
    quad2d_centred<G>(yv, 10, aM, aG, d);
#pragma unroll
    for (int j = 0; j < kQuadOut; ++j) rmg[j] = ll2f(d[j]) * im[j] * ig[j];
    quad2d_centred<G>(yv, 2, sv, aM, d);
#pragma unroll
    for (int j = 0; j < kQuadOut; ++j)
      rum[j] = ll2f(d[j]) * div_ftz(P.sig_scale, sg[j]) * im[j];
    quad2d_centred<G>(yv, 4, sv, aG, d);
    unsigned slow = 0;
#pragma unroll
    for (int j = 0; j < kQuadOut; ++j) {
      const float rug = ll2f(d[j]) * div_ftz(P.sig_scale, sg[j]) * ig[j];
      const float den = 1.0f - rmg[j] * rmg[j];
      const bool jm = km >> j & 1, jg = kg >> j & 1;
      // fused_solve's expression with its contractions written out
      float r2 = div_ftz(__fmaf_rn(-__fmul_rn(2.0f * rum[j], rug), rmg[j],
                                   __fmaf_rn(rum[j], rum[j], __fmul_rn(rug, rug))),
                         den);
      r2 = jm ? (jg ? r2 : rum[j] * rum[j]) : (jg ? rug * rug : 0.0f);
      float v = sg[j] * r2;
      if (!(v > 0.0f) || isinf(v)) v = 0.0f;
      if (sg[j] > 0.0f) {
        ms[j] = v;
        if (jm && jg && !(den > 1e-3f)) slow |= 1u << j;
      }
    }
    // nearly collinear columns: the general solve from the limbs summed afresh
#pragma unroll
    for (int j = 0; j < kQuadOut; ++j) {
      if (slow >> j & 1) {
        int L[kLimbs];
#pragma unroll
        for (int k = 0; k < kLimbs; ++k) {
          L[k] = 0;
#pragma unroll 1
          for (int i = 0; i < G::W; ++i) L[k] += yv[(size_t)k * G::PY + j + i];
        }
        ms[j] = fused_measure<2, R>(P, sg[j], sv[j], L);
      }
      acc_m += __float2int_rn(ms[j] * P.sum_scale);
    }
  }
  if (out_measure) {
#pragma unroll
    for (int j = 0; j < kQuadOut; ++j)
      if (j < rows) out_measure[(size_t)(yr + j) * P.vx + x] = ms[j];
  }
  return acc_m;
}

template <int WND, typename T, int TY, int R>
__global__ void __launch_bounds__(Quad2D<TY, R>::NT, Quad2D<TY, R>::CTAS)
    k_quad2d(const T* __restrict__ mov, const T* __restrict__ Ust, const float* __restrict__ sig,
             const int* __restrict__ su, FusedParams P, const Xform* __restrict__ xf, int k0,
             unsigned long long* __restrict__ acc, float* __restrict__ out_measure) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ TileShared T_;
  const int slot = blockIdx.x;
  long long m = quad_tile_2d<WND, T, T, TY, R>(mov, Ust, sig, su, P, xf + k0 + slot, blockIdx.y,
                                               smem_raw, T_, slot == 0 ? out_measure : nullptr);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m += __shfl_down_sync(0xffffffffu, m, o);
  if ((threadIdx.x & 31) == 0 && threadIdx.x < Quad2D<TY, R>::ST)
    atomicAdd(acc + 2 * (size_t)(k0 + slot), (unsigned long long)m);
}

template <int WND, typename T, int R, int TY>
cudaError_t quad2d_launch_rt(const FusedLaunch& L) {
  using G = Quad2D<TY, R>;
  if (L.P.kbits != PatchConst<2, R>::K || L.P.n != PatchConst<2, R>::N)
    return cudaErrorInvalidValue;
  auto kern = k_quad2d<WND, T, TY, R>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)G::BYTES);
  if (e != cudaSuccess) return e;
  FusedParams P = L.P;
  P.ntx = (P.vx + 31) / 32;
  dim3 grid(L.cnt, P.ntx * ((P.vy + TY - 1) / TY));
  kern<<<grid, G::NT, G::BYTES, L.stream>>>((const T*)L.mov, (const T*)L.ust, L.sig, L.su, P, L.xf,
                                            L.k0, L.acc, L.out_measure);
  return cudaGetLastError();
}

}  // namespace lc2
