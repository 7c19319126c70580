// lc2_quad_fixed.cuh -- k_fused_quad's scheme for a resampled ultrasound
// (HighResolutionModality: Fixed).
#pragma once

#include "lc2_fused_fixed.cuh"
#include "lc2_quad.cuh"

namespace lc2 {

// Square root of x in [1, 2^64) from y = rsqrt.approx(x): one Newton step on
// the exact residual x - (x y)^2 (Markstein 1990), which rounds as sqrtf does
// (compared on every float of that range).
__device__ __forceinline__ float sqrt_from(float x, float y) {
  const float g = __fmul_rn(x, y);
  return __fmaf_rn(__fmaf_rn(-g, g, x), 0.5f * y, g);
}

// Per transform the ultrasound's window sums change, those of the static MR/CT
// and its Sobel magnitude do not (FixedStatic): eight limbs per point (S_U,
// invalid count, UU, UM, UG), no Sobel of the warped image, and the static
// sums and solve factors read per output voxel. Quads, planes, passes and
// hand-over as in k_fused_quad, except that the moments warps, which have
// registers to spare here, also run the x pass (with it in the solve warps:
// 3.78 ms below); the leaving slice's (2 qU + invalid, qM, qG) come from a ring
// of 16-byte entries that only their thread touches. The solve is
// solve_centred_static's, in the same float operations.
//
// Bound by the solve warps' serial chain (the moments and x pass alone take
// 2.0 ms). 160^3, radius 3, 50 transforms: moments 3.73 ms on 16-row tiles of
// one point per thread -> 2.58 (sqrtf instead of sqrt_from: 2.73), with the
// resampling 4.44 -> 3.11 ms. Two solving groups on alternate slices would need
// 24 warps at 80 registers, where the moments warps spill (3.93).
template <int TY, int R>
__global__ void __launch_bounds__(QuadGeom<TY, R, kFixedLimbs, 3, false>::NT, 1)
    k_fixed_quad(const float* __restrict__ Ub, const int* __restrict__ Mq,
                 const int* __restrict__ Gq, FixedStatic F, QuadParams Q, int k0,
                 unsigned long long* __restrict__ acc) {
  using G = QuadGeom<TY, R, kFixedLimbs, 3, false>;
  using C = PatchConst<3, R>;
  constexpr int KB = C::K;
  constexpr unsigned kmask = (1u << KB) - 1u;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const FusedParams& P = Q.f;
  quad_start();
  // the window / solve warps first, as in k_fused_quad
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
    const float* Us = Ub + (size_t)slot * Q.volume;
    const int off = Q.origin + (y0 - R + 4 * q) * Q.px + x0 - R + hx;
    unsigned o4[4];  // byte offsets in a slice
#pragma unroll
    for (int i = 0; i < 4; ++i) o4[i] = 4u * (unsigned)(off + i * Q.px);
    int* a = A + hx * G::YP + 4 * q;
    int4* ring = reinterpret_cast<int4*>(smem_raw) + tid;
#pragma unroll
    for (int k = 0; k < 3 * G::RING; ++k) ring[k * G::PT] = make_int4(0, 0, 0, 0);
    int sU[4], sI[4];
    long long s[4][3];  // UU, UM, UG
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      sU[i] = sI[i] = 0;
#pragma unroll
      for (int k = 0; k < 3; ++k) s[i][k] = 0;
    }
    auto at = [&](auto* p, int e) { return p + (long long)e * (long long)Q.slice; };
    // lines of the slices ahead, one L2 prefetch per warp and slice: the
    // image's, rows of the warp's quad, 3 lines
    const unsigned po = 4u * (unsigned)(Q.origin + (y0 - R + 4 * min(tid >> 5, G::NQ - 1) + lane / 3) *
                                                       Q.px + x0 - R + 32 * (lane % 3));
    const bool pf = tid < 32 * G::NQ && lane < 12 && lane % 3 * 32 < G::HX + 31;
    const int e_end = min(ze + R, P.vz);
    auto prefetch = [&](int e) {
      if (pf && e < e_end) prefetch_l2(reinterpret_cast<const char*>(at(Us, e)) + po);
    };
#pragma unroll
    for (int k = 0; k < kQuadAhead; ++k) prefetch(e0 + 1 + k);
    // the entering slice's fields, loaded a slice ahead
    float un[4];
    int mn[4], gn[4];
    auto load = [&](int e) {
      const float* pu = at(Us, e);
      const int *pm = at(Mq, e), *pg = at(Gq, e);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        un[i] = ld_off(pu, o4[i]);
        mn[i] = ld_off(pm, o4[i]);
        gn[i] = ld_off(pg, o4[i]);
      }
    };
    load(e0);
    // x-pass job of this thread: (column part, limb, quad of rows)
    const bool xjob = tid < G::XP * G::XJOBS;
    const int xpart = tid / G::XJOBS, xj = tid - xpart * G::XJOBS, xl = xj / G::NQ;
    const int xc = min(xpart * G::XC, 32 - G::XC) * G::YP + 4 * (xj - xl * G::NQ);
    const int* xa = A + (xjob ? xl * G::PA + xc : 0);
    int* xy = Y + (xjob ? xl * G::PY + xc : 0);
    int rs = 0;
    for (int e = e0; e < ze + R; ++e) {
      prefetch(e + 1 + kQuadAhead);
      int4* rg = ring + rs * 3 * G::PT;
      rs = rs + 1 == G::RING ? 0 : rs + 1;
      const int4 lu = rg[0], lm = rg[G::PT], lg = rg[2 * G::PT];
      const int pl[4] = {lu.x, lu.y, lu.z, lu.w}, ml[4] = {lm.x, lm.y, lm.z, lm.w},
                gl[4] = {lg.x, lg.y, lg.z, lg.w};
      int pn[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int qu = quant(un[i], P.qu), inv = (un[i] > 1e-6f) ? 0 : 1;
        pn[i] = 2 * qu + inv;
        const int ql = pl[i] >> 1, du = qu - ql;
        sU[i] += du;
        sI[i] += inv - (pl[i] & 1);
        s[i][0] += (long long)du * (qu + ql);
        s[i][1] += (long long)qu * mn[i];
        s[i][1] += (long long)(-ql) * ml[i];
        s[i][2] += (long long)qu * gn[i];
        s[i][2] += (long long)(-ql) * gl[i];
      }
      rg[0] = make_int4(pn[0], pn[1], pn[2], pn[3]);
      rg[G::PT] = make_int4(mn[0], mn[1], mn[2], mn[3]);
      rg[2 * G::PT] = make_int4(gn[0], gn[1], gn[2], gn[3]);
      load(min(e + 1, P.vz + R));
      const int z = e - R;
      if (z >= zb) {
        bar_sync_n<4, G::PT>();  // the x pass has read the last slice's limbs
        if (own) {
          *reinterpret_cast<int4*>(a) = make_int4(sU[0], sU[1], sU[2], sU[3]);
          *reinterpret_cast<int4*>(a + G::PA) = make_int4(sI[0], sI[1], sI[2], sI[3]);
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            *reinterpret_cast<int4*>(a + (2 + 2 * k) * G::PA) =
                make_int4((int)((unsigned)s[0][k] & kmask), (int)((unsigned)s[1][k] & kmask),
                          (int)((unsigned)s[2][k] & kmask), (int)((unsigned)s[3][k] & kmask));
            *reinterpret_cast<int4*>(a + (3 + 2 * k) * G::PA) =
                make_int4((int)(s[0][k] >> KB), (int)(s[1][k] >> KB), (int)(s[2][k] >> KB),
                          (int)(s[3][k] >> KB));
          }
        }
        bar_sync_n<1, G::PT>();              // limbs of slice z written
        if (z > zb) bar_sync_n<3, G::NT>();  // the last slice's patch sums are read
        quad_xpass<G>(xjob, xa, xy);
        bar_arrive_n<2, G::NT>();            // x sums of slice z written
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
  const unsigned go = (unsigned)yr * P.vx + x;               // of the first in a slice
  unsigned o8[kQuadOut];                                     // byte offsets of (S_M, S_G)
#pragma unroll
  for (int j = 0; j < kQuadOut; ++j) o8[j] = 8u * (go + j * P.vx);
  long long acc_m = 0, acc_s = 0;
  // static sums and solve factors of the slice, loaded a slice ahead
  int2 nsm[kQuadOut];
  float4 nsv[kQuadOut];
  auto load_static = [&](int z) {
#pragma unroll
    for (int j = 0; j < kQuadOut; ++j) {
      if (z < ze && j < rows) {
        nsm[j] = ld_off(F.s + (size_t)z * plane, o8[j]);
        nsv[j] = ld_off(F.sv + (size_t)z * plane, 2u * o8[j]);
      }
    }
  };
#pragma unroll
  for (int j = 0; j < kQuadOut; ++j) {
    nsm[j] = make_int2(0, 0);
    nsv[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  }
  load_static(zb);
  const int* yv = Y + (size_t)lane * G::YP + row0;
  // what the solve of a slice keeps of its patch sums
  float fuu[kQuadOut], rum[kQuadOut], rug[kQuadOut], psv[kQuadOut][3], sg[kQuadOut];
#pragma unroll
  for (int j = 0; j < kQuadOut; ++j) {
    fuu[j] = 0.0f;
    rum[j] = rug[j] = sg[j] = 0.0f;
    psv[j][0] = psv[j][1] = psv[j][2] = 0.0f;
  }
  // measure and weighting factor of each output from them (fuu = 0: none)
  auto finish = [&]() {
#pragma unroll
    for (int j = 0; j < kQuadOut; ++j) {
      const float iu = rsqrt_ftz(fuu[j]), sigma = sqrt_from(fuu[j], iu) * P.sig_scale;
      const float im = psv[j][0], ig = psv[j][1], rmg = psv[j][2];
      const float um = rum[j] * iu * im, ug = rug[j] * iu * ig;
      const float den = 1.0f - rmg * rmg;
      const bool jm = im > 0.0f, jg = ig > 0.0f;
      float r2 = div_ftz(__fmaf_rn(-__fmul_rn(2.0f * um, ug), rmg,
                                   __fmaf_rn(um, um, __fmul_rn(ug, ug))),
                         den);
      r2 = jm ? (jg ? r2 : um * um) : (jg ? ug * ug : 0.0f);
      float m = sigma * r2;
      if (!(m > 0.0f) || isinf(m)) m = 0.0f;
      if (fuu[j] > 0.0f) {
        acc_m += __float2int_rn(m * P.sum_scale);
        acc_s += __float2int_rn(sigma * P.sum_scale);
      }
    }
  };
  for (int z = zb; z < ze; ++z) {
    finish();
    int2 sm[kQuadOut];
#pragma unroll
    for (int j = 0; j < kQuadOut; ++j) {
      sm[j] = nsm[j];
      psv[j][0] = nsv[j].x;
      psv[j][1] = nsv[j].y;
      psv[j][2] = nsv[j].z;
    }
    load_static(z + 1);
    bar_sync_n<2, G::NT>();  // x sums of slice z written
    {
      int aU[kQuadOut], aI[kQuadOut], aS[kQuadOut];
      long long duu[kQuadOut], d[kQuadOut], du2[kQuadOut];
      quad_window<G>(yv, aU);
      quad_window<G>(yv + G::PY, aI);
      quad_centred<G>(yv, 2, aU, aU, duu);
#pragma unroll
      for (int j = 0; j < kQuadOut; ++j) aS[j] = sm[j].x;
      quad_centred<G>(yv, 4, aU, aS, d);
#pragma unroll
      for (int j = 0; j < kQuadOut; ++j) aS[j] = sm[j].y;
      quad_centred<G>(yv, 6, aU, aS, du2);
#pragma unroll
      for (int j = 0; j < kQuadOut; ++j) {
        bool ok = j < rows && aI[j] == 0 && duu[j] > P.thr_var;
        rum[j] = ll2f(d[j]);
        rug[j] = ll2f(du2[j]);
        const float den = 1.0f - psv[j][2] * psv[j][2];
        if (ok && psv[j][0] > 0.0f && psv[j][1] > 0.0f && !(den > 1e-3f)) {
          // nearly collinear columns: the double solve
          float sigma, m;
          solve_centred_static(duu[j], d[j], du2[j],
                               make_float4(psv[j][0], psv[j][1], psv[j][2], 0.0f), F.d, F.nv,
                               (size_t)z * plane + (go + j * P.vx), P.thr_var, P.sig_scale, sigma, m);
          acc_m += __float2int_rn(m * P.sum_scale);
          acc_s += __float2int_rn(sigma * P.sum_scale);
          ok = false;
        }
        fuu[j] = ok ? ll2f(duu[j]) : 0.0f;
      }
    }
    if (z + 1 < ze) bar_arrive_n<3, G::NT>();  // they may be overwritten
  }
  finish();
  fixed_flush(acc_m, acc_s, acc + 2 * (size_t)(k0 + slot));
  quad_join();
}

template <int R>
cudaError_t fixed_quad_launch_r(const FixedLaunch& L, const int* q, const PadLayout& lay,
                                const QuadPlan& plan) {
  using G24 = QuadGeom<24, R, kFixedLimbs, 3, false>;
  using G16 = QuadGeom<16, R, kFixedLimbs, 3, false>;
  if (L.P.kbits != PatchConst<3, R>::K || L.P.n != PatchConst<3, R>::N)
    return cudaErrorInvalidValue;
  const float* pre = L.pre + lay.first();
  const int *qm = q + lay.first(), *qg = q + lay.volume() + lay.first();
  return quad_launches(
      L.P, lay, plan, L.cnt,
      [&](const QuadParams& Q, dim3 grid) {
        return quad_launch_one(k_fixed_quad<24, R>, grid, G24::NT, G24::BYTES, L.stream, false, pre, qm,
                               qg, L.S, Q, L.k0, L.acc);
      },
      [&](const QuadParams& Q, dim3 grid) {
        return quad_launch_one(k_fixed_quad<16, R>, grid, G16::NT, G16::BYTES, L.stream, true, pre, qm,
                               qg, L.S, Q, L.k0, L.acc);
      });
}

// The moments pass of a group of presampled ultrasounds (padded layout); q:
// the quantised static image and its Sobel magnitude, padded, one after the
// other. Defined in lc2_quad_fixed.cu.
cudaError_t fixed_quad_launch(const FixedLaunch& L, const int* q, const PadLayout& lay,
                              const QuadPlan& plan);

}  // namespace lc2
