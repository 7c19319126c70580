// The kernels' short forms of math functions against the functions, bit for bit,
// over the ranges that they are used on. Prints the number of arguments that
// differ for each.
#include <cstdio>
#include <cstring>

#include "../../lc2registration_gb300/csrc/lc2_quad_fixed.cuh"

__device__ unsigned long long g_bad[5];

// Every float whose bits lie in [first, last).
template <typename F>
__global__ void k_each(unsigned first, unsigned last, int which, F differs) {
  unsigned long long n = 0;
  for (unsigned long long b = first + blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; b < last;
       b += (unsigned long long)gridDim.x * blockDim.x)
    n += differs(__uint_as_float((unsigned)b));
  if (n) atomicAdd(&g_bad[which], n);
}

struct Sqrt {
  __device__ bool operator()(float x) const {
    return __float_as_uint(lc2::sqrt_from(x, lc2::rsqrt_ftz(x))) != __float_as_uint(sqrtf(x));
  }
};
struct Rsqrt {
  __device__ bool operator()(float x) const {
    return __float_as_uint(lc2::rsqrt_ftz(x)) != __float_as_uint(rsqrtf(x));
  }
};
struct Floor {
  __device__ static bool one(float q) {
    unsigned n;
    float r;
    lc2::floor_split(q, n, r);
    const float f = floorf(q);
    return (int)(n - lc2::kFloorBias) != (int)f || !(r == q - f);
  }
  __device__ bool operator()(float q) const { return one(q) || one(-q); }
};
struct Div {  // denominators; numerators of the size of a product of correlations
  __device__ bool operator()(float b) const {
    bool bad = false;
    for (float a = 1.9999f; a > 1e-30f; a *= 0.0137f)
      bad = bad || __float_as_uint(lc2::div_ftz(a, b)) != __float_as_uint(__fdividef(a, b)) ||
            __float_as_uint(lc2::div_ftz(-a, b)) != __float_as_uint(__fdividef(-a, b));
    return bad;
  }
};
struct DivScale {  // weighting factors; their scale over them is in [2^-32, 1]
  __device__ bool operator()(float b) const {
    bool bad = false;
    for (float t = 1.0f; t > 2e-10f; t *= 0.0317f)
      bad = bad || __float_as_uint(lc2::div_ftz(b * t, b)) != __float_as_uint(__fdividef(b * t, b));
    return bad;
  }
};

static unsigned bits(float f) {
  unsigned u;
  memcpy(&u, &f, 4);
  return u;
}

int main() {
  const unsigned one = bits(1.0f), two64 = bits(18446744073709551616.0f);
  k_each<<<1216, 256>>>(one, two64, 0, Sqrt());
  k_each<<<1216, 256>>>(one, two64, 1, Rsqrt());
  k_each<<<1216, 256>>>(0u, bits(4194304.0f), 2, Floor());
  k_each<<<1216, 256>>>(bits(1e-3f), one + 1, 3, Div());
  k_each<<<1216, 256>>>(bits(1e-3f), bits(1e30f), 4, DivScale());
  unsigned long long bad[5];
  cudaError_t e = cudaMemcpyFromSymbol(bad, g_bad, sizeof(bad));
  if (e != cudaSuccess) {
    std::printf("%s\n", cudaGetErrorString(e));
    return 1;
  }
  std::printf("sqrt %llu rsqrt %llu floor %llu div %llu divscale %llu\n", bad[0], bad[1], bad[2], bad[3], bad[4]);
  return 0;
}
