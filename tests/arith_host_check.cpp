// Host build of the device arithmetic (erdos-strauss_gb300/csrc/es_arith.cuh) for the CPU tests: 2^64 mod n
// and the Montgomery constants against 128-bit arithmetic, over all sizes of n and the edges of the
// float quotient's ranges. Built so that a signed overflow ends the program.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <random>
#define __device__
#define __forceinline__ inline
#define __constant__
static inline unsigned long long __umul64hi(unsigned long long a, unsigned long long b) {
  return (unsigned long long)(((unsigned __int128)a * b) >> 64);
}
static inline int __ffsll(long long x) { return x ? __builtin_ctzll((unsigned long long)x) + 1 : 0; }
static inline int __clzll(long long x) { return x ? __builtin_clzll((unsigned long long)x) : 64; }
static inline unsigned atomicOr(unsigned *p, unsigned v) { const unsigned o = *p; *p |= v; return o; }
#include "es_arith.cuh"
using namespace es;

static bool check(u64 n) {
  const unsigned __int128 R = (unsigned __int128)1 << 64;
  const Mont M = mont_init(n);
  const u64 one = (u64)(R % n), r2 = (u64)((unsigned __int128)one * one % n);
  if (M.one == one && M.r2 == r2 && M.ninv * n == ~0ull) return true;
  printf("FAIL n=%llu: one %llu for %llu, r2 %llu for %llu\n", n, M.one, one, M.r2, r2);
  return false;
}

int main() {
  std::mt19937_64 g(0xA217);
  const u64 T = 1ull << 63, edges[] = {3, 1ull << 32, 1ull << 40, 1ull << 62, T, T / 3 * 4, T + (T >> 1), ~0ull - 99};
  for (u64 e : edges)
    for (u64 k = 0; k < 50; ++k)
      if (!check((e + 2 * k) | 1) || (e > 200 && !check((e - 2 * k) | 1))) return 1;
  for (int t = 0; t < 400000; ++t) {
    const u64 n = (g() >> (t % 62)) | 1;
    if (n > 1 && !check(n)) return 1;
  }
  for (int t = 0; t < 100000; ++t)                     // between 2^63 and 4/3 2^63, where 10^19 lies
    if (!check((T + g() % (T / 3)) | 1)) return 1;
  return 0;
}
