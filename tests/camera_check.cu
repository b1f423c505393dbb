// The camera sample's raster and wavelength expressions (df32.cuh) against
// float64's, rounded: random, central and edge coordinates of many widths.
// Prints one line a function: name, inputs, mismatches.
#include <cstdio>

#include "df32.cuh"

using namespace vmr;

__device__ unsigned long long mix(unsigned long long z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__global__ void check(unsigned long long n, unsigned long long* bad) {
  const unsigned widths[] = {1u, 2u, 3u, 77u, 640u, 1280u, 4095u, 4096u, 5000u, 65537u, (1u << 22) - 1u, 1u << 22};
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const unsigned long long r = mix(i + 1), t = mix(r);
    const unsigned w = widths[r % 12];
    const unsigned long long top = (unsigned long long)(w < 4096u ? w : 4096u) << 40, mid = (unsigned long long)w << 39;
    unsigned long long k = t % top;
    switch (r >> 60 & 7u) {
      case 0: k = (mid < top ? mid : 0) + (t >> 40) % 65u; break;
      case 1: k = (mid < top ? mid : top) - (t >> 40) % 65u; break;
      case 2: k = (t >> 40) % 65u; break;
      case 3: k = top - 1 - (t >> 40) % 65u; break;
      case 4: k = (k >> 38 << 38) + (t & 1u); break;
      default: break;
    }
    if (k >= top) k = top - 1;
    if (__float_as_uint(raster_ndc(k, w)) != __float_as_uint(raster_ndc64(k, w))) atomicAdd(bad, 1ull);
    unsigned long long v = t >> 12;
    if ((r >> 60 & 7u) == 0) v = (v & 0xffull) << 44;
    if ((r >> 60 & 7u) == 1) v >>= (r >> 30 & 31u);
    if ((r >> 60 & 7u) == 2) v = (1ull << 52) - 1 - (v & 0xffull);
    if (__float_as_uint(wavelength52(v)) != __float_as_uint(wavelength64(v))) atomicAdd(bad + 1, 1ull);
  }
}

int main() {
  unsigned long long *d, h[2] = {}, n = 1ull << 28;
  if (cudaMalloc(&d, sizeof(h)) != cudaSuccess || cudaMemset(d, 0, sizeof(h)) != cudaSuccess) return 1;
  check<<<1216, 256>>>(n, d);
  if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
  printf("raster_ndc %llu %llu\nwavelength %llu %llu\n", n, h[0], n, h[1]);
  return 0;
}
