// What the device headers need to compile for the host: vector types, the intrinsics
// that one thread can answer, and declarations of those it cannot (never called).
#pragma once
#include <cstdint>

#define __constant__
#define __noinline__ __attribute__((noinline))
struct uint2 {
  uint32_t x, y;
};
struct alignas(16) uint4 {
  uint32_t x, y, z, w;
};
struct alignas(16) ulonglong2 {
  unsigned long long x, y;
};
inline uint4 make_uint4(uint32_t x, uint32_t y, uint32_t z, uint32_t w) { return {x, y, z, w}; }
inline ulonglong2 make_ulonglong2(unsigned long long x, unsigned long long y) { return {x, y}; }
inline uint32_t __funnelshift_l(uint32_t lo, uint32_t hi, uint32_t shift) {
  shift &= 31;
  return shift ? (hi << shift) | (lo >> (32 - shift)) : hi;
}
uint32_t __shfl_xor_sync(uint32_t, uint32_t, int);
uint64_t __shfl_sync(uint32_t, uint64_t, uint32_t);
void __syncwarp();
uint64_t __ldcg(const uint64_t*);
struct HostThread {
  uint32_t x;
};
static const HostThread threadIdx = {0};
