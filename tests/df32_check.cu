// Every float32 input of the functions in df32.cuh against CUDA's float64
// functions rounded, and random and edge pairs of the QMC fractions for the
// two-argument ones.  Prints one line a function: name, inputs, mismatches.
#include <cstdio>

#include "df32.cuh"

using namespace vmr;
enum Fn { kSin, kCos, kSinCosS, kSinCosC, kAcos, kAtan, kOverPi };

__device__ bool same(float a, float b) {
  return __float_as_uint(a) == __float_as_uint(b) || (isnan(a) && isnan(b));
}

template <int F>
__global__ void all_floats(unsigned long long lo, unsigned long long hi, unsigned long long* bad) {
  unsigned long long n = 0;
  for (unsigned long long u = lo + blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; u < hi;
       u += (unsigned long long)gridDim.x * blockDim.x) {
    const float x = __uint_as_float((unsigned)u);
    float a, b, c;
    if (F == kSin) { a = sin_rn(x); b = (float)sin((double)x); }
    if (F == kCos) { a = cos_rn(x); b = (float)cos((double)x); }
    if (F == kSinCosS) { sincos_rn(x, a, c); b = (float)sin((double)x); }
    if (F == kSinCosC) { sincos_rn(x, c, a); b = (float)cos((double)x); }
    if (F == kAcos) { a = acos_rn(x); b = (float)acos((double)x); }
    if (F == kAtan) { a = atan_rn(x); b = (float)atan((double)x); }
    if (F == kOverPi) { a = over_pi(x); b = (float)((double)x / 3.14159265358979323846); }
    if (!same(a, b)) ++n;
  }
  if (n) atomicAdd(bad, n);
}

__device__ unsigned long long mix(unsigned long long z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
// A fraction's bits: uniform, or close to a multiple of 1/8, or small.
__device__ unsigned long long frac(unsigned long long i, int which) {
  const unsigned long long r = mix(i * 2 + which + 1), k = r >> 12;
  switch (r & 7u) {
    case 0: return (k & 0x7ull) << 49;
    case 1: return (((k & 0x7ull) << 49) + (r >> 40 & 0xffu)) & (kOne52 - 1);
    case 2: return (((k & 0x7ull) << 49) - (r >> 40 & 0xffu)) & (kOne52 - 1);
    case 3: return k >> (r >> 3 & 31u);
    default: return k;
  }
}
__global__ void pairs(unsigned long long n, unsigned long long* bad) {
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const unsigned long long k0 = frac(i, 0), k1 = frac(i, 1);
    float x, y, z, X, Y, Z, a, b, A, B;
    cosine_hemisphere(k0, k1, x, y, z);
    cosine_hemisphere64(k0, k1, X, Y, Z);
    if (!same(x, X) || !same(y, Y) || !same(z, Z)) atomicAdd(bad, 1ull);
    triangle_uv(k0, k1, a, b);
    triangle_uv64(k0, k1, A, B);
    if (!same(a, A) || !same(b, B)) atomicAdd(bad + 1, 1ull);
    if (!same(frac52(k0), (float)((double)k0 / 4503599627370496.0))) atomicAdd(bad + 2, 1ull);
  }
}

int main() {
  unsigned long long* d;
  cudaMalloc(&d, 64);
  auto report = [&](const char* name, unsigned long long n, int k) {
    unsigned long long h[8] = {};
    const cudaError_t e = cudaMemcpy(h, d, 64, cudaMemcpyDeviceToHost);
    printf("%s %llu %llu\n", name, n, e == cudaSuccess ? h[k] : ~0ull);
  };
  auto run = [&](auto kernel, const char* name, unsigned top) {  // all floats of magnitude bits <= top, both signs
    for (unsigned s = 0; s < 2; ++s) {
      cudaMemset(d, 0, 64);
      const unsigned long long lo = (unsigned long long)s << 31;
      kernel<<<152 * 16, 128>>>(lo, lo + top + 1, d);
      report(name, top + 1ull, 0);
    }
  };
  const unsigned f16 = 0x41800000u, one = 0x3f800000u, nan = 0x7fc00001u;
  run(all_floats<kSin>, "sin", f16);
  run(all_floats<kCos>, "cos", f16);
  run(all_floats<kSinCosS>, "sincos.s", f16);
  run(all_floats<kSinCosC>, "sincos.c", f16);
  run(all_floats<kAcos>, "acos", one);
  run(all_floats<kAtan>, "atan", nan);
  run(all_floats<kOverPi>, "over_pi", 0x40000000u);
  cudaMemset(d, 0, 64);
  const unsigned long long n = 1ull << 27;
  pairs<<<152 * 16, 128>>>(n, d);
  report("cosine_hemisphere", n, 0);
  report("triangle_uv", n, 1);
  report("frac52", n, 2);
  return cudaDeviceSynchronize() == cudaSuccess ? 0 : 1;
}
