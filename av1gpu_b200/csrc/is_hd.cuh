// is_hd.cuh - arithmetic compiled for the device and, by the CPU tests, for the host: the qualifiers, and the CUDA integer
// intrinsics' host forms where no CUDA compiler provides them.
#pragma once
#include <stdint.h>
#include <type_traits>

#ifdef __CUDACC__
#define IS_HD __host__ __device__ __forceinline__   // called on both sides
#define IS_DEV __device__ __forceinline__            // the device's, and the tests' host build's
#else
#define IS_HD static inline
#define IS_DEV static inline
#include <string.h>
#include <algorithm>
#include <cstdlib>
using std::abs;
using std::max;
using std::min;
static inline uint32_t __umulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
static inline int __clz(int v) { return v ? __builtin_clz((unsigned)v) : 32; }
static inline int __ffs(int v) { return __builtin_ffs(v); }
static inline int __ffsll(long long v) { return __builtin_ffsll(v); }
static inline uint32_t __float_as_uint(float f) { uint32_t u; memcpy(&u, &f, 4); return u; }
static inline float __uint_as_float(uint32_t u) { float f; memcpy(&f, &u, 4); return f; }
#endif
