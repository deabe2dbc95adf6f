// Stand-in for CUDA's header, found before it when tests compile device code
// for the host (emulate.h): the types and the few functions that the kernels
// under test use.
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#define __device__
#define __host__
#define __global__
#define __shared__
#define __forceinline__ inline
#define __launch_bounds__(...)
#define __align__(x) __attribute__((aligned(x)))

struct double2 { double x, y; };
struct float2 { float x, y; };
struct double4 { double x, y, z, w; };
struct float4 { float x, y, z, w; };
inline double2 make_double2(double x, double y) { return {x, y}; }
inline float2 make_float2(float x, float y) { return {x, y}; }
inline double4 make_double4(double x, double y, double z, double w) { return {x, y, z, w}; }
inline float4 make_float4(float x, float y, float z, float w) { return {x, y, z, w}; }

inline double __dmul_rn(double a, double b) { return a * b; }
inline float __fmul_rn(float a, float b) { return a * b; }
inline double __fma_rn(double a, double b, double c) { return fma(a, b, c); }
inline float __fmaf_rn(float a, float b, float c) { return fmaf(a, b, c); }
inline double __ddiv_rn(double a, double b) { return a / b; }
inline float __fdiv_rn(float a, float b) { return a / b; }
inline double __dadd_rn(double a, double b) { return a + b; }
inline double __dsub_rn(double a, double b) { return a - b; }
template <class T>
T __shfl_down_sync(unsigned, T, int);  // declared only: no kernel under test exchanges by it
template <class T>
T __ldcg(const T *p) { return *p; }

struct emu_dim3 { unsigned x, y, z; };
extern emu_dim3 threadIdx, blockIdx, blockDim, gridDim;
void emu_barrier(bool block);
inline void __syncthreads() { emu_barrier(true); }
inline void __syncwarp(unsigned = 0xffffffffu) { emu_barrier(false); }
void emu_copy16(void *dst, const void *src);
void emu_copies_wait();
