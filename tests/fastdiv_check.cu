// fastdiv_check.cu -- the operations of FastDiv (positive denominators, square
// root; hormone_b200/csrc/hmn_div.cuh) against IEEE division and square root on
// the GPU: whatever is not flagged must have the same bits, the sign of a zero
// included.
//
//   fastdiv_check N SEED     N operands per family; one line
//                            "<family> n=<n> flagged=<n> mismatches=<n>" each,
//                            exit status 1 on any mismatch.
//
// Quotients: random; at the range limits; long runs of ones or zeros; a = +-0;
// a next to b; a/b next to a rounding midpoint; both significands within a few
// units of 2.  Radicands: random; at the range limits; next to the square of a
// number, and of a midpoint between two; the two significands that lie closest
// to a midpoint (1 + 2^-52 and 4 - 2^-51) over every exponent.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>

#include "hmn_div.cuh"

__device__ __forceinline__ uint64_t mix(uint64_t x) {
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}
__device__ double from(uint64_t sign, int e, uint64_t mant) {
  return __longlong_as_double((long long)((sign << 63) | ((uint64_t)(e + 1023) << 52) | (mant & 0xfffffffffffffull)));
}
__device__ double nudge(double x, int k) { return __longlong_as_double(__double_as_longlong(x) + k); }
__device__ uint64_t runs(uint64_t m, uint64_t r) {
  const int len = (int)(r % 52) + 1, at = (int)((r >> 8) % 52);
  const uint64_t run = (((1ull << len) - 1) << at) & 0xfffffffffffffull;
  return (r >> 20) & 1 ? m | run : m & ~run;
}

__global__ void check(int fam, long long n, uint64_t seed, unsigned long long* bad, unsigned long long* flagged,
                      double* ex) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    const uint64_t r0 = mix(seed + 3 * (uint64_t)t), r1 = mix(r0), r2 = mix(r1);
    const uint64_t s = r2 & 1;
    bool flag = false;
    double a, b, got, want, y = 0.0, yw = 0.0;
    if (fam < 7) {
      a = from(s, (int)(r2 >> 8) % 40 - 20 + 0, r0);
      b = from(0, (int)((r2 >> 20) % 41) - 20, r1);
      if (fam == 0) {
        a = from(s, (int)((r2 >> 8) % 1041) - 520, r0);
        b = from(0, (int)((r2 >> 24) % 1041) - 520, r1);
      } else if (fam == 1) {
        a = from(s, (int)((r2 >> 8) % 8) - 4 + ((r2 >> 16) & 1 ? 500 : -500), r0);
        b = from((r2 >> 40) & 1, (int)((r2 >> 24) % 8) - 4 + ((r2 >> 32) & 1 ? 500 : -500), r1);
      } else if (fam == 2) {
        a = from(s, 0, runs(r0, r2 >> 8));
        b = from(0, 0, runs(r1, r2 >> 30));
      } else if (fam == 3) {
        a = s ? -0.0 : 0.0;
      } else if (fam == 4) {
        a = nudge(b, (int)(r2 >> 8) % 9 - 4) * (s ? -1.0 : 1.0);
      } else if (fam == 5) {  // a = b (q + u/2) rounded, and its neighbours
        const double q = from(0, 0, r0);
        b = from(0, 0, r1);
        a = nudge(__fma_rn(b, 0x1p-53, b * q), (int)((r2 >> 8) % 3) - 1);
      } else {
        a = from(s, 0, 0xfffffffffffffull - (r0 % 64));
        b = from(0, 0, 0xfffffffffffffull - (r1 % 64));
      }
      y = hmn::recip_pos(b, flag);
      got = hmn::div_pos(a, b, y, flag);
      want = a / b;
      yw = 1.0 / b;
    } else {
      b = 0.0;
      const int e = (int)((r2 >> 8) % 1041) - 520;
      if (fam == 7) {
        a = from(0, e, r0);
      } else if (fam == 8) {
        a = from((r2 >> 50) & 1, (int)((r2 >> 8) % 8) - 4 + ((r2 >> 16) & 1 ? 500 : -500), r0);
      } else if (fam == 9) {
        const double z = from(0, (int)((r2 >> 8) % 400) - 200, r0);
        a = nudge(z * z, (int)((r2 >> 40) % 5) - 2);
      } else if (fam == 10) {  // (z + u/2)^2
        const double z = from(0, 0, r0);
        a = nudge(__fma_rn(z, z, z * 0x1p-52), (int)((r2 >> 40) % 5) - 2);
      } else {
        a = (t & 1) ? from(0, 2 * (int)((t >> 1) % 500) - 500, 1) : from(0, 2 * (int)((t >> 1) % 500) - 499, ~0ull);
      }
      got = hmn::sqrt_pos(a, flag);
      want = sqrt(a);
    }
    if (flag) {
      atomicAdd(flagged, 1ull);
    } else if (__double_as_longlong(got) != __double_as_longlong(want) ||
               __double_as_longlong(y) != __double_as_longlong(yw)) {
      if (atomicAdd(bad, 1ull) == 0) {
        ex[0] = a;
        ex[1] = b;
        ex[2] = got;
        ex[3] = want;
      }
    }
  }
}

int main(int argc, char** argv) {
  const long long n = argc > 1 ? atoll(argv[1]) : (1ll << 24);
  const uint64_t seed = argc > 2 ? strtoull(argv[2], nullptr, 10) : 1;
  unsigned long long* d;
  double* ex;
  if (cudaMalloc(&d, 16) != cudaSuccess || cudaMalloc(&ex, 32) != cudaSuccess) return 2;
  const char* names[12] = {"div_random", "div_limits", "div_runs", "div_zero", "div_nearly_equal", "div_midpoints",
                           "div_near_two", "sqrt_random", "sqrt_limits", "sqrt_squares", "sqrt_midpoints",
                           "sqrt_closest"};
  int fail = 0;
  for (int f = 0; f < 12; f++) {
    cudaMemset(d, 0, 16);
    check<<<148 * 8, 256>>>(f, n, seed + 0x9e3779b9ull * f, d, d + 1, ex);
    unsigned long long h[2];
    double e[4];
    if (cudaMemcpy(h, d, 16, cudaMemcpyDeviceToHost) != cudaSuccess ||
        cudaMemcpy(e, ex, 32, cudaMemcpyDeviceToHost) != cudaSuccess) {
      fprintf(stderr, "kernel failed: %s\n", cudaGetErrorString(cudaGetLastError()));
      return 2;
    }
    printf("%s n=%lld flagged=%llu mismatches=%llu\n", names[f], n, h[1], h[0]);
    if (h[0]) {
      printf("  e.g. a=%a b=%a fast=%a ieee=%a\n", e[0], e[1], e[2], e[3]);
      fail = 1;
    }
  }
  return fail;
}
