// The branch-free roots and quotient of jf_device.cuh against the general
// operations, bit for bit: test_gpu_mid_range.py compiles and runs this file.
#include "jf_device.cuh"

struct Found {
  unsigned long long n;  // operands that differ
  float a, b;            // one of them
};

namespace {

__device__ void note(Found* f, float a, float b) {
  if (atomicAdd(&f->n, 1ull) == 0ull) {
    f->a = a;
    f->b = b;
  }
}

__device__ bool same(float x, float y) { return __float_as_uint(x) == __float_as_uint(y); }

// operands with the bit patterns first .. first + n - 1
__global__ void roots(uint32_t first, uint32_t n, Found* f) {
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const float a = __uint_as_float(first + k);
    float h;
    if (!same(jf_sqrt_mid(a, &h), sqrtf(a))) note(f, a, 0.0f);
    if (!same(jf_inv_sqrt_mid(a), 1.0f / sqrtf(a))) note(f + 1, a, 0.0f);
  }
}

__device__ uint32_t mix(uint64_t z) {  // splitmix64 (Steele, Lea and Flood 2014)
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return (uint32_t)((z ^ (z >> 31)) >> 32);
}

// Every mantissa of the divisor at exponent de, with numerators no larger: the
// powers of two, the divisor's and all-ones mantissas and their neighbours at a
// few exponents, and `random` random ones.
__global__ void quotients(int de, int random, uint64_t seed, Found* f) {
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < (1u << 23); k += gridDim.x * blockDim.x) {
    const uint32_t db = ((uint32_t)(de + 127) << 23) | k;
    const float d = __uint_as_float(db);
    auto check = [&](float n) {
      if (!(fabsf(n) <= d) || fabsf(n) < 1e-5f) return;
      if (!same(jf_div_mid(n, d), n / d)) note(f, n, d);
      if (!same(jf_div_mid(n, -d), n / -d)) note(f, n, -d);
    };
    for (int ne = de - 3; ne <= de; ++ne) {
      const uint32_t e = (uint32_t)(ne + 127) << 23;
      for (int j = -2; j <= 2; ++j) {
        check(__uint_as_float(e + j));      // about a power of two
        check(__uint_as_float((e | k) + j));  // about the divisor's mantissa
        check(__uint_as_float((e | (k ^ 0x7fffffu)) + j));
      }
    }
    for (int r = 0; r < random; ++r) {
      const uint32_t u = mix(seed + ((uint64_t)k << 20) + r);
      const uint32_t e = (uint32_t)(de - (int)(u >> 27) % 16 + 127) << 23;
      check(__uint_as_float(e | (u & 0x7fffffu)));
    }
  }
}

}  // namespace

// out[3]: roots, reciprocal roots, quotients; 0 or a CUDA error
extern "C" int mid_range(Found* out, int random) {
  Found* f;
  cudaError_t err = cudaMalloc(&f, 3 * sizeof(Found));
  if (err != cudaSuccess) return (int)err;
  cudaMemset(f, 0, 3 * sizeof(Found));
  // every operand of 2^-60 .. 2^60
  for (int e = -60; e < 60; ++e) roots<<<1184, 256>>>((uint32_t)(e + 127) << 23, 1u << 23, f);
  for (int de : {-17, -16, -1, 0, 1, 10, 29, 30}) quotients<<<1184, 256>>>(de, random, 77 + de, f + 2);
  err = cudaMemcpy(out, f, 3 * sizeof(Found), cudaMemcpyDeviceToHost);
  cudaFree(f);
  return (int)err;
}
