// lc2_quad.cuh -- the 3D moments pass on presampled images, in column quads.
#pragma once

#include "lc2_fused.cuh"
#include "lc2_quad_plan.hpp"

namespace lc2 {

struct QuadParams {
  FusedParams f;
  int px;                 // row pitch of the padded images
  int origin;             // offset of voxel (0, 0) in a padded slice
  size_t slice, volume;   // strides of the padded images
  int y0;                 // first output row of the launch's tiles
};

// The launches of a plan: the second one starts as SMs come free from the first
// (programmatic dependent launch; both only read what earlier launches wrote
// and add to the same sums) and its last CTA waits for the first one's end, so
// that the second's end is the end of both.
template <typename L24, typename L16>
cudaError_t quad_launches(const FusedParams& f, const PadLayout& lay, const QuadPlan& plan, int cnt,
                          L24 l24, L16 l16) {
  QuadParams Q;
  Q.f = f;
  Q.px = lay.px;
  Q.origin = (int)lay.origin();
  Q.slice = lay.slice();
  Q.volume = lay.volume();
  Q.f.ntx = (f.vx + 31) / 32;
  Q.f.zchunk = plan.z24;
  Q.y0 = 0;
  auto grid = [&](int rows) {
    return dim3(cnt, Q.f.ntx * rows, (f.vz + Q.f.zchunk - 1) / Q.f.zchunk);
  };
  cudaError_t e = l24(Q, grid(plan.rows24));
  if (e != cudaSuccess || !plan.rows16) return e;
  Q.f.zchunk = plan.z16;
  Q.y0 = 24 * plan.rows24;
  return l16(Q, grid(plan.rows16));
}

// One launch of kern; after: it may start before the launch before it is done.
template <typename... KP, typename... A>
cudaError_t quad_launch_one(void (*kern)(KP...), dim3 grid, int threads, size_t smem,
                            cudaStream_t stream, bool after, A... args) {
  cudaError_t e =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = after ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

// At the start of a CTA of 24-row tiles: the next launch may fill SMs as they
// come free. At the end of one of 16-row tiles: the launch's last CTA stays
// until the launch before it is done.
__device__ __forceinline__ void quad_start() {
  asm volatile("griddepcontrol.launch_dependents;");
}
__device__ __forceinline__ void quad_join() {
  if (blockIdx.x == gridDim.x - 1 && blockIdx.y == gridDim.y - 1 && blockIdx.z == gridDim.z - 1)
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// ---- moments ----
// The moments pass of a resampled MR/CT on presampled images (radius 1-4, the
// default): for each of its 32 x TY output tiles a CTA marches along z as
// k_fused does -- Sobel magnitude of the entering slice, exact z-window sums of
// the twelve limbs at every halo point, window passes, solve -- with the same
// integers and float operations, so the same bits. What it does differently:
//
// * A moments thread owns a quad, four rows of one halo column, with all its
//   window sums in registers. Its four Sobel magnitudes share one 6 x 3
//   neighbourhood (18 64-bit reads instead of 36) and its limbs leave as
//   128-bit stores; the planes are [column][row] with a row pitch of an odd
//   number of quads, so stores along columns and reads along rows are free of
//   bank conflicts.
// * The x window pass reads and writes 128 bits (four rows of a limb) per step,
//   from the limb planes A to the planes Y; the y windows need no pass: a
//   solving thread reads the three quads around its four output rows and sums
//   them in registers.
// * Moments warps and window / solve warps run side by side, handing A over
//   through named barriers: the moments of slice z+1 overlap the x pass and
//   solve of slice z. The last part of a slice's solve (its divisions) needs
//   no shared memory and is written after the next slice's hand-over, where the
//   compiler mixes it with the next windows' reads.
// * The images have zero borders (PadLayout), so no load has a bounds test,
//   and each moments warp prefetches its rows into L2 kQuadAhead slices ahead:
//   a slice takes about 2 us, hardly more than a DRAM access under load
//   (without the prefetch 6.7 ms instead of 5.85 below).
//
// Bound: the data pipe of shared memory and L1 (82 % of its peak; about 2900
// wavefronts of 3600 cycles per slice of a tile at radius 4). The register file
// sets the shape: 16 warps at 128 registers; 20 warps would need 96, and the
// moments warps' window sums spill there. The previous kernel (one halo point
// per thread with its limbs as 32-bit words, y pass and solve as phases of
// their own on 24 warps) took 1752 M shared-memory wavefronts for 19 transforms
// at 256^3 against 1308 M and 603 instructions per voxel against 402.
// 256^3, radius 4, f16, 19 transforms: 8.31 -> 5.85 ms of moments (437 -> 308 us
// per transform); 128^3 -> 96^3 radius 3, 100 transforms: 2606 -> 1890 us with
// the resampling. Tried and slower at 256^3: eight output rows per solving
// thread (13.9 ms: three warps cannot hide the reads), the x pass by the moments
// warps (8.1), the Sobel magnitudes as a pass of their own (7.5 and 0.7 for the
// pass); both tile heights in one kernel (5.99, more spills); one CTA per SM
// with an equal share of all columns (2.7 us per slice instead of 1.9: the
// halos of neighbouring tiles come from DRAM when they march at different z).
constexpr int kQuadOut = 4;  // output rows per solving thread

// NL limb planes; NRING 16-byte ring entries per moments thread and slice of
// the window; SOBEL: the (Sz, Dz) planes of a resampled MR/CT.
template <int TY, int R, int NL = kLimbs, int NRING = 1, bool SOBEL = true>
struct QuadGeom {
  static constexpr int R_ = R, W = 2 * R + 1;
  static constexpr int HX = 32 + 2 * R, HY = TY + 2 * R;
  static constexpr int NQ = (HY + 3) / 4;                     // halo quads per column
  static constexpr int TAIL = 2 * R * NQ;                     // threads of the columns beyond 32
  static constexpr int PWARPS = NQ + (TAIL + 31) / 32;        // moments warps
  static constexpr int PT = 32 * PWARPS;
  static constexpr int CT = 32 * (TY / kQuadOut);             // window / solve threads
  static constexpr int NT = PT + CT;
  // x pass: jobs (limb, quad of rows), their 32 output columns in XP parts
  static constexpr int XJOBS = NL * NQ;
  static constexpr int XT = SOBEL ? CT : PT;                  // threads that run the x pass
  static constexpr int XP = XT / XJOBS > 3 ? 3 : XT / XJOBS > 0 ? XT / XJOBS : 1;
  static constexpr int XC = (32 + XP - 1) / XP;
  // (Sz, Dz) planes: the halo with a one-voxel margin. Pitch = 2 mod 4 float2,
  // so that the 8-column tail's four quads of a warp (rows 4 apart) read
  // distinct banks.
  static constexpr int SP = HX + 2 + (6 - (HX + 2) % 4) % 4;
  static constexpr int SR = 4 * NQ + 2;
  static constexpr int NM = 2 * (HX + 2) + 2 * (4 * NQ);      // margin points
  // limb planes [column][row]: row pitch an odd number of quads
  static constexpr int YP = 4 * (NQ | 1);
  // plane strides: consecutive (limb, quad) jobs of the x pass on consecutive
  // 16-byte bank groups
  static constexpr int PA = HX * YP + (32 + 4 * (NQ % 8) - HX * YP % 32) % 32;
  static constexpr int PY = 32 * YP + (32 + 4 * (NQ % 8) - 32 * YP % 32) % 32;
  static constexpr int RING = 2 * R + 1;
  static constexpr size_t OFF_SD = sizeof(int4) * (size_t)NRING * RING * PT;  // after the ring
  static constexpr size_t OFF_A = OFF_SD + (SOBEL ? sizeof(float2) * 2 * (size_t)SP * SR : 0);
  static constexpr size_t OFF_Y = OFF_A + sizeof(int) * (size_t)NL * PA;
  static constexpr size_t BYTES = OFF_Y + sizeof(int) * (size_t)NL * PY;
  static constexpr int NV = (kQuadOut + W - 1 + 3) / 4;       // quads a solving thread reads
  static_assert(SP % 4 == 2 && SP >= HX + 2 && OFF_A % 16 == 0 && PA % 4 == 0 && PY % 4 == 0, "");
  static_assert(TY % kQuadOut == 0 && TY / 4 - kQuadOut / 4 + NV <= NQ, "a solve stays in the plane");
  static_assert(NM <= PT, "one margin point per moments thread");
  static_assert(XJOBS <= XT, "every x job has a thread");
  static_assert(BYTES <= 227 * 1024, "one CTA's shared memory must fit an SM");
};

template <int ID, int N>
__device__ __forceinline__ void bar_sync_n() {
  asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(N) : "memory");
}
template <int ID, int N>
__device__ __forceinline__ void bar_arrive_n() {
  asm volatile("bar.arrive %0, %1;" ::"n"(ID), "n"(N) : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}
// Load at a 32-bit byte offset from a pointer that is the same for the CTA.
template <typename T>
__device__ __forceinline__ T ld_off(const T* p, unsigned off) {
  return __ldg(reinterpret_cast<const T*>(reinterpret_cast<const char*>(p) + off));
}
constexpr int kQuadAhead = 4;  // slices that L2 prefetches run ahead of the loads

// rsqrtf and __fdividef without their denormal handling: the arguments are
// integers >= 1, weighting factors > 1e-3 and denominators in (1e-3, 1], for
// which both give the same bits.
__device__ __forceinline__ float rsqrt_ftz(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float div_ftz(float a, float b) {
  float r;
  asm("div.approx.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// Window sums of one limb at kQuadOut consecutive rows: o[j] = sum of rows
// j .. j + 2R of the column at y.
template <typename G>
__device__ __forceinline__ void quad_window(const int* __restrict__ y, int* o) {
  int v[4 * G::NV];
#pragma unroll
  for (int i = 0; i < G::NV; ++i) {
    const int4 c = reinterpret_cast<const int4*>(y)[i];
    v[4 * i] = c.x;
    v[4 * i + 1] = c.y;
    v[4 * i + 2] = c.z;
    v[4 * i + 3] = c.w;
  }
  int a = 0;
#pragma unroll
  for (int i = 0; i < G::W; ++i) a += v[i];
  o[0] = a;
#pragma unroll
  for (int j = 1; j < kQuadOut; ++j) {
    a += v[j + G::W - 1] - v[j - 1];
    o[j] = a;
  }
}

// Centred sums D = n S - a b of kQuadOut outputs, S = hi 2^K + lo from the
// window sums of limb planes L (lo) and L + 1 (hi); n 2^K fits 31 bits by the
// choice of K.
template <typename G>
__device__ __forceinline__ void quad_centred(const int* __restrict__ y, int L, const int* a,
                                             const int* b, long long* d) {
  using C = PatchConst<3, G::R_>;
  constexpr int n = (int)C::N, nk = (int)(C::N << C::K);
  int lo[kQuadOut], hi[kQuadOut];
  quad_window<G>(y + (size_t)L * G::PY, lo);
  quad_window<G>(y + (size_t)(L + 1) * G::PY, hi);
#pragma unroll
  for (int j = 0; j < kQuadOut; ++j)
    d[j] = (long long)hi[j] * nk + (long long)lo[j] * n - (long long)a[j] * b[j];
}

// x window pass from the limb planes to Y: four rows of one limb per thread, a
// running sum along XC + 2R columns.
template <typename G>
__device__ __forceinline__ void quad_xpass(bool job, const int* __restrict__ a,
                                           int* __restrict__ y) {
  if (G::XP * G::XJOBS == G::XT || job) {
    int4 v[G::XC + G::W - 1];
    int4 w = make_int4(0, 0, 0, 0);
#pragma unroll
    for (int i = 0; i < G::XC + G::W - 1; ++i) {
      v[i] = *reinterpret_cast<const int4*>(a + i * G::YP);
      if (i < G::W) {
        w.x += v[i].x;
        w.y += v[i].y;
        w.z += v[i].z;
        w.w += v[i].w;
      } else {
        w.x += v[i].x - v[i - G::W].x;
        w.y += v[i].y - v[i - G::W].y;
        w.z += v[i].z - v[i - G::W].z;
        w.w += v[i].w - v[i - G::W].w;
      }
      if (i >= G::W - 1) *reinterpret_cast<int4*>(y + (i - G::W + 1) * G::YP) = w;
    }
  }
}

// One output voxel with nearly collinear columns the general way: its limbs
// summed afresh from the planes.
template <int TY, int R>
__device__ __forceinline__ float quad_measure_slow(const FusedParams& P, const int* y, float sg,
                                                   int su) {
  using G = QuadGeom<TY, R>;
  int L[kLimbs];
#pragma unroll
  for (int k = 0; k < kLimbs; ++k) L[k] = 0;
#pragma unroll 1
  for (int i = 0; i < G::W; ++i) {
#pragma unroll
    for (int k = 0; k < kLimbs; ++k) L[k] += y[(size_t)k * G::PY + i];
  }
  return fused_measure<3, R>(P, sg, su, L);
}

template <int TY, int R>
__global__ void __launch_bounds__(QuadGeom<TY, R>::NT, 1)
    k_fused_quad(const float* __restrict__ Mb, const int* __restrict__ Uq,
                 const int2* __restrict__ Ss, QuadParams Q, int k0,
                 unsigned long long* __restrict__ acc, float* __restrict__ out_measure) {
  using G = QuadGeom<TY, R>;
  using C = PatchConst<3, R>;
  constexpr int KB = C::K;
  constexpr unsigned kmask = (1u << KB) - 1u;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const FusedParams& P = Q.f;
  if constexpr (TY == 24) quad_start();
  // the window / solve warps come first: theirs is the longer chain, and the
  // schedulers prefer lower warps (5.81 against 6.03 ms below)
  const int tid = (int)threadIdx.x < G::CT ? threadIdx.x + G::PT : threadIdx.x - G::CT;
  const int lane = tid & 31, slot = blockIdx.x, tile = blockIdx.y;
  const int x0 = (tile % P.ntx) * 32, y0 = Q.y0 + (tile / P.ntx) * TY;
  const int zb = blockIdx.z * P.zchunk;
  const int ze = min(zb + P.zchunk, P.vz);
  const int e0 = zb - R;
  int* A = reinterpret_cast<int*>(smem_raw + G::OFF_A);
  int* Y = reinterpret_cast<int*>(smem_raw + G::OFF_Y);

  if (tid < G::PT) {
    // ---- moments: one quad of four rows of one halo column per thread ----
    int hx, q;
    if (tid < 32 * G::NQ) {
      hx = lane;
      q = tid >> 5;
    } else {
      const int t = tid - 32 * G::NQ;
      q = t / (2 * R);
      hx = 32 + t - q * (2 * R);
    }
    const bool own = tid < 32 * G::NQ || tid - 32 * G::NQ < G::TAIL;
    if (!own) {  // idle lanes follow along on the last quad; they write nothing
      q = G::NQ - 1;
      hx = 32 + 2 * R - 1;
    }
    const float* Ms = Mb + (size_t)slot * Q.volume;
    const int off = Q.origin + (y0 - R + 4 * q) * Q.px + x0 - R + hx;
    unsigned o4[4];  // byte offsets in a slice
#pragma unroll
    for (int i = 0; i < 4; ++i) o4[i] = 4u * (unsigned)(off + i * Q.px);
    // margin point of this thread: (row, column) of the (Sz, Dz) plane
    int mr, mcx;
    {
      const int m = tid < G::NM ? tid : 0;
      if (m < 2 * (G::HX + 2)) {
        mr = m < G::HX + 2 ? 0 : G::SR - 1;
        mcx = m < G::HX + 2 ? m : m - (G::HX + 2);
      } else {
        const int t = m - 2 * (G::HX + 2);
        mr = 1 + (t >> 1);
        mcx = (t & 1) ? G::HX + 1 : 0;
      }
    }
    const unsigned om = 4u * (unsigned)(Q.origin + (y0 - R - 1 + mr) * Q.px + x0 - R - 1 + mcx);
    const bool margin = tid < G::NM;
    const int sm = mr * G::SP + mcx;
    const int sd = (4 * q + 1) * G::SP + hx + 1;  // plane index of the quad's first point
    const int a_off = hx * G::YP + 4 * q;
    int sM[4], sG[4];
    long long s[4][5];  // UM, UG, MM, GG, MG
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      sM[i] = sG[i] = 0;
#pragma unroll
      for (int k = 0; k < 5; ++k) s[i][k] = 0;
    }
    int4* ring = reinterpret_cast<int4*>(smem_raw) + tid;
    float2* SD = reinterpret_cast<float2*>(smem_raw + G::OFF_SD);
#pragma unroll
    for (int k = 0; k < G::RING; ++k) ring[k * G::PT] = make_int4(0, 0, 0, 0);
    auto slice_m = [&](int e) { return Ms + (long long)e * (long long)Q.slice; };
    auto slice_u = [&](int e) { return Uq + (long long)e * (long long)Q.slice; };
    // lines of the slices ahead, one L2 prefetch per warp and slice: lanes
    // 0-11 the image, 12-23 the ultrasound; rows of the warp's quad, 3 lines
    const int pl = lane < 12 ? lane : lane - 12;
    const unsigned po = 4u * (unsigned)(Q.origin + (y0 - R + 4 * min(tid >> 5, G::NQ - 1) + pl / 3) * Q.px +
                                        x0 - R + 32 * (pl % 3));
    const bool pf = tid < 32 * G::NQ && lane < 24 && pl % 3 * 32 < G::HX + 31;
    const int e_end = min(ze + R, P.vz);
    auto prefetch = [&](int e) {
      if (pf && e < e_end) {
        if (lane < 12)
          prefetch_l2(reinterpret_cast<const char*>(slice_m(e)) + po);
        else
          prefetch_l2(reinterpret_cast<const char*>(slice_u(e)) + po);
      }
    };
    // M of slices e, e+1 and e+2 (prefetched) at the quad and the margin point
    float m0[4], m1[4], m2[4], g0, g1, g2;
    auto planes = [&](float2* dst, const float* a, const float* b, const float* c, float am,
                      float bm, float cm) {
      if (own) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          dst[sd + i * G::SP] = make_float2(a[i] + 2.0f * b[i] + c[i], c[i] - a[i]);
      }
      if (margin) dst[sm] = make_float2(am + 2.0f * bm + cm, cm - am);
    };
    {
      float mp[4], gp;
      const float *pa = slice_m(e0 - 1), *pb = slice_m(e0), *pc = slice_m(e0 + 1),
                  *pd = slice_m(e0 + 2);
#pragma unroll
      for (int k = 0; k < kQuadAhead; ++k) prefetch(e0 + 3 + k);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        mp[i] = ld_off(pa, o4[i]);
        m0[i] = ld_off(pb, o4[i]);
        m1[i] = ld_off(pc, o4[i]);
        m2[i] = ld_off(pd, o4[i]);
      }
      gp = ld_off(pa, om);
      g0 = ld_off(pb, om);
      g1 = ld_off(pc, om);
      g2 = ld_off(pd, om);
      planes(SD, mp, m0, m1, gp, g0, g1);
    }
    // entering ultrasound, leaving M and ultrasound, loaded a slice ahead; a
    // slice that no window holds yet leaves as zeros (the border slice)
    int un[4], ul[4];
    float ml[4];
    auto load_next = [&](int e) {
      const int l = e - 2 * R - 1;
      const int lz = l >= e0 ? l : -R - 1;
      const int* pu = slice_u(e);
      const int* pl = slice_u(lz);
      const float* pm = slice_m(lz);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        un[i] = ld_off(pu, o4[i]);
        ul[i] = ld_off(pl, o4[i]);
        ml[i] = ld_off(pm, o4[i]);
      }
    };
    load_next(e0);
    int rs = 0, buf = 0;
    for (int e = e0; e < ze + R; ++e) {
      prefetch(e + 3 + kQuadAhead);
      bar_sync_n<1, G::PT>();  // planes(e) written; planes(e-1) read
      const float2* S = SD + buf * (G::SP * G::SR) + sd;
      // Sobel magnitudes of the four points from the 6 x 3 neighbourhood, in
      // the order of operations of fused_sobel_sd
      int qg[4];
      {
        float rd[6], tz[6], sl[6], sc[6], sr[6];
#pragma unroll
        for (int j = 0; j < 6; ++j) {
          const float2 a = S[(j - 1) * G::SP - 1], b = S[(j - 1) * G::SP],
                       c = S[(j - 1) * G::SP + 1];
          rd[j] = c.x - a.x;
          tz[j] = a.y + 2.0f * b.y + c.y;
          sl[j] = a.x;
          sc[j] = b.x;
          sr[j] = c.x;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float gx = rd[i] + 2.0f * rd[i + 1] + rd[i + 2];
          const float gy = (sl[i + 2] - sl[i]) + 2.0f * (sc[i + 2] - sc[i]) + (sr[i + 2] - sr[i]);
          const float gz = tz[i] + 2.0f * tz[i + 1] + tz[i + 2];
          qg[i] = quant(sqrt_approx(gx * gx + gy * gy + gz * gz), P.qg);
        }
      }
      // planes(e+1) from M(e), M(e+1), M(e+2)
      buf ^= 1;
      planes(SD + buf * (G::SP * G::SR), m0, m1, m2, g0, g1, g2);
      const int4 gl4 = ring[rs * G::PT];
      ring[rs * G::PT] = make_int4(qg[0], qg[1], qg[2], qg[3]);
      rs = rs + 1 == G::RING ? 0 : rs + 1;
      const int gl[4] = {gl4.x, gl4.y, gl4.z, gl4.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int qm = quant(m0[i], P.qm), qml = quant(ml[i], P.qm);
        const int qu = un[i], nul = -ul[i], ngl = -gl[i];
        const int dm = qm - qml, dg = qg[i] + ngl;
        sM[i] += dm;
        sG[i] += dg;
        s[i][0] += (long long)qu * qm;
        s[i][0] += (long long)nul * qml;
        s[i][1] += (long long)qu * qg[i];
        s[i][1] += (long long)nul * gl[i];
        s[i][2] += (long long)dm * (qm + qml);
        s[i][3] += (long long)dg * (qg[i] + gl[i]);
        s[i][4] += (long long)qm * qg[i];
        s[i][4] += (long long)qml * ngl;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        m0[i] = m1[i];
        m1[i] = m2[i];
      }
      g0 = g1;
      g1 = g2;
      {
        const float* pd = slice_m(min(e + 3, P.vz + R + 1));
#pragma unroll
        for (int i = 0; i < 4; ++i) m2[i] = ld_off(pd, o4[i]);
        g2 = ld_off(pd, om);
      }
      load_next(min(e + 1, P.vz + R));
      const int z = e - R;
      if (z >= zb) {
        if (z > zb) bar_sync_n<3, G::NT>();  // the x pass has read the last slice's limbs
        if (own) {
          int* a = A + a_off;
          *reinterpret_cast<int4*>(a) = make_int4(sM[0], sM[1], sM[2], sM[3]);
          *reinterpret_cast<int4*>(a + G::PA) = make_int4(sG[0], sG[1], sG[2], sG[3]);
#pragma unroll
          for (int k = 0; k < 5; ++k) {
            *reinterpret_cast<int4*>(a + (2 + 2 * k) * G::PA) =
                make_int4((int)((unsigned)s[0][k] & kmask), (int)((unsigned)s[1][k] & kmask),
                          (int)((unsigned)s[2][k] & kmask), (int)((unsigned)s[3][k] & kmask));
            *reinterpret_cast<int4*>(a + (3 + 2 * k) * G::PA) =
                make_int4((int)(s[0][k] >> KB), (int)(s[1][k] >> KB), (int)(s[2][k] >> KB),
                          (int)(s[3][k] >> KB));
          }
        }
        bar_arrive_n<2, G::NT>();  // limbs of slice z written
      }
    }
    return;
  }

  // ---- window sums and solve: kQuadOut rows of one column per thread ----
  const int ct = tid - G::PT;
  const int row0 = kQuadOut * (ct >> 5);
  const int x = x0 + lane, yr = y0 + row0;
  const size_t plane = (size_t)P.vx * P.vy;
  const int rows = x < P.vx ? min(kQuadOut, P.vy - yr) : 0;  // output rows in the grid
  const size_t g_off = (size_t)yr * P.vx + x;
  long long acc_m = 0;
  // x-pass job of this thread: (column part, limb, quad of rows)
  const bool xjob = ct < G::XP * G::XJOBS;
  const int xpart = ct / G::XJOBS, xj = ct - xpart * G::XJOBS, xl = xj / G::NQ;
  const int xc = min(xpart * G::XC, 32 - G::XC) * G::YP + 4 * (xj - xl * G::NQ);
  const int *xa = A + (xjob ? xl * G::PA + xc : 0);
  int* xy = Y + (xjob ? xl * G::PY + xc : 0);
  // weighting factor and S_U of the slice, loaded two slices ahead; zero
  // outside the grid
  const unsigned so = 8u * (unsigned)(Q.origin + yr * Q.px + x);
  auto slice_s = [&](int z) { return Ss + (long long)z * (long long)Q.slice; };
  int2 s1[kQuadOut], s2[kQuadOut];
#pragma unroll
  for (int j = 0; j < kQuadOut; ++j) {
    s1[j] = ld_off(slice_s(zb), so + j * 8u * Q.px);
    s2[j] = ld_off(slice_s(zb + 1), so + j * 8u * Q.px);
  }
  const int* yv = Y + (size_t)lane * G::YP + row0;
  bar_sync_n<2, G::NT>();  // limbs of slice zb written
  quad_xpass<G>(xjob, xa, xy);
  if (zb + 1 < ze) bar_arrive_n<3, G::NT>();  // the limbs may be overwritten
  bar_sync_n<4, G::CT>();                     // the x sums of slice zb are complete
  // what the solve of a slice keeps of its patch sums
  float im[kQuadOut], ig[kQuadOut], rmg[kQuadOut], fum[kQuadOut], fug[kQuadOut], psg[kQuadOut];
  float ms[kQuadOut];
  unsigned km = 0, kg = 0, slow = 0;
#pragma unroll
  for (int j = 0; j < kQuadOut; ++j) im[j] = ig[j] = rmg[j] = fum[j] = fug[j] = psg[j] = ms[j] = 0.0f;
  // the measures of slice z from them
  auto finish = [&](int z) {
    float m[kQuadOut];
#pragma unroll
    for (int j = 0; j < kQuadOut; ++j) {
      const float iu = div_ftz(P.sig_scale, psg[j]);  // 1 / sqrt(D_uu)
      const float rum = fum[j] * iu * im[j], rug = fug[j] * iu * ig[j];
      const float den = 1.0f - rmg[j] * rmg[j];
      const bool jm = km >> j & 1, jg = kg >> j & 1;
      // fused_solve's expression with its contractions written out
      float r2 = div_ftz(__fmaf_rn(-__fmul_rn(2.0f * rum, rug), rmg[j],
                                   __fmaf_rn(rum, rum, __fmul_rn(rug, rug))),
                         den);
      r2 = jm ? (jg ? r2 : rum * rum) : (jg ? rug * rug : 0.0f);
      float v = psg[j] * r2;
      if (!(v > 0.0f) || isinf(v)) v = 0.0f;
      m[j] = psg[j] > 0.0f ? ((slow >> j & 1) ? ms[j] : v) : 0.0f;
      acc_m += __float2int_rn(m[j] * P.sum_scale);
    }
    if (out_measure && slot == 0 && z >= zb) {
#pragma unroll
      for (int j = 0; j < kQuadOut; ++j)
        if (j < rows) out_measure[(size_t)z * plane + g_off + (size_t)j * P.vx] = m[j];
    }
  };
  for (int z = zb; z < ze; ++z) {
    finish(z - 1);
    int sv[kQuadOut];
#pragma unroll
    for (int j = 0; j < kQuadOut; ++j) {
      psg[j] = __int_as_float(s1[j].x);
      sv[j] = s1[j].y;
      s1[j] = s2[j];
      s2[j] = ld_off(slice_s(min(z + 2, P.vz)), so + j * 8u * Q.px);
    }
    {
      int aM[kQuadOut], aG[kQuadOut];
      long long d[kQuadOut];
      km = kg = slow = 0;
      quad_window<G>(yv, aM);
      quad_window<G>(yv + G::PY, aG);
      quad_centred<G>(yv, 6, aM, aM, d);
#pragma unroll
      for (int j = 0; j < kQuadOut; ++j) {
        if (d[j] > P.thr_m) km |= 1u << j;
        im[j] = rsqrt_ftz(ll2f(d[j]));
      }
      quad_centred<G>(yv, 8, aG, aG, d);
#pragma unroll
      for (int j = 0; j < kQuadOut; ++j) {
        if (d[j] > P.thr_g) kg |= 1u << j;
        ig[j] = rsqrt_ftz(ll2f(d[j]));
      }
      quad_centred<G>(yv, 10, aM, aG, d);
#pragma unroll
      for (int j = 0; j < kQuadOut; ++j) {
        rmg[j] = ll2f(d[j]) * im[j] * ig[j];
        const float den = 1.0f - rmg[j] * rmg[j];
        if (psg[j] > 0.0f && ((km & kg) >> j & 1) && !(den > 1e-3f)) slow |= 1u << j;
      }
      quad_centred<G>(yv, 2, sv, aM, d);
#pragma unroll
      for (int j = 0; j < kQuadOut; ++j) fum[j] = ll2f(d[j]);
      quad_centred<G>(yv, 4, sv, aG, d);
#pragma unroll
      for (int j = 0; j < kQuadOut; ++j) fug[j] = ll2f(d[j]);
      if (slow) {
#pragma unroll 1
        for (int j = 0; j < kQuadOut; ++j) {
          float sj = 0.0f;
          int vj = 0;
#pragma unroll
          for (int i = 0; i < kQuadOut; ++i)
            if (i == j) {
              sj = psg[i];
              vj = sv[i];
            }
          const float v = (slow >> j & 1) ? quad_measure_slow<TY, R>(P, yv + j, sj, vj) : 0.0f;
#pragma unroll
          for (int i = 0; i < kQuadOut; ++i)
            if (i == j) ms[i] = v;
        }
      }
    }
    if (z + 1 < ze) {
      bar_sync_n<4, G::CT>();  // the patch sums of slice z are read
      bar_sync_n<2, G::NT>();  // limbs of slice z+1 written
      quad_xpass<G>(xjob, xa, xy);
      if (z + 2 < ze) bar_arrive_n<3, G::NT>();  // the limbs may be overwritten
      bar_sync_n<4, G::CT>();                    // the x sums of slice z+1 are complete
    }
  }
  finish(ze - 1);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc_m += __shfl_down_sync(0xffffffffu, acc_m, o);
  if (lane == 0) atomicAdd(acc + 2 * (size_t)(k0 + slot), (unsigned long long)acc_m);
  if constexpr (TY != 24) quad_join();
}

template <int R>
cudaError_t quad_launch_r(const FusedLaunch& L, const float* M, const int* uq, const int2* ss,
                          const PadLayout& lay, const QuadPlan& plan) {
  if (L.P.kbits != PatchConst<3, R>::K || L.P.n != PatchConst<3, R>::N)
    return cudaErrorInvalidValue;
  M += lay.first();
  uq += lay.first();
  ss += lay.first();
  return quad_launches(
      L.P, lay, plan, L.cnt,
      [&](const QuadParams& Q, dim3 grid) {
        return quad_launch_one(k_fused_quad<24, R>, grid, QuadGeom<24, R>::NT, QuadGeom<24, R>::BYTES,
                               L.stream, false, M, uq, ss, Q, L.k0, L.acc, L.out_measure);
      },
      [&](const QuadParams& Q, dim3 grid) {
        return quad_launch_one(k_fused_quad<16, R>, grid, QuadGeom<16, R>::NT, QuadGeom<16, R>::BYTES,
                               L.stream, true, M, uq, ss, Q, L.k0, L.acc, L.out_measure);
      });
}

// The moments pass of a group of presampled images (padded layout). Defined in
// lc2_quad.cu.
cudaError_t quad_launch(const FusedLaunch& L, const float* M, const int* uq, const int2* ss,
                        const PadLayout& lay, const QuadPlan& plan);

}  // namespace lc2
