// Two fp32 numbers an instruction (sm_100a's packed fp32 arithmetic: the same roundings as two scalar operations).
#pragma once
#include <stdint.h>

typedef unsigned long long Pair;
__device__ __forceinline__ Pair pair_of(uint32_t a, uint32_t b) { Pair v; asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(a), "r"(b)); return v; }
__device__ __forceinline__ Pair pair_of(float a, float b) { return pair_of(__float_as_uint(a), __float_as_uint(b)); }
__device__ __forceinline__ Pair pair_fma(Pair a, Pair b, Pair c) { Pair v; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c)); return v; }
__device__ __forceinline__ Pair pair_mul(Pair a, Pair b) { Pair v; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b)); return v; }
__device__ __forceinline__ Pair pair_add(Pair a, Pair b) { Pair v; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b)); return v; }
__device__ __forceinline__ float pair_at(Pair v, int i) { uint32_t a, b; asm("mov.b64 {%0, %1}, %2;" : "=r"(a), "=r"(b) : "l"(v)); return __uint_as_float(i ? b : a); }
