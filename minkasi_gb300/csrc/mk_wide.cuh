// 32-byte streaming loads and stores (sm_100 and later), addresses 32-byte
// aligned.  A warp whose lanes each hold 8 consecutive doubles touches 16 lines
// per 16-byte load, whatever it takes of them: the L1's tag stage, not its data
// path, bounds such a stream, and half as many instructions halve that.
#pragma once
#include <stdint.h>

namespace mk {

__host__ __device__ __forceinline__ bool aligned32(const void *p) { return (uintptr_t)p % 32 == 0; }

__device__ __forceinline__ void ld32(const double *p, double *v) {  // 4 values
  asm volatile("ld.global.cs.v4.f64 {%0, %1, %2, %3}, [%4];"
               : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3])
               : "l"(p));
}
__device__ __forceinline__ void ld32(const float *p, float *v) {  // 8 values
  asm volatile("ld.global.cs.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
               : "l"(p));
}
__device__ __forceinline__ void ld32(const int32_t *p, int32_t *v) {  // 8 values
  asm volatile("ld.global.cs.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "l"(p));
}
__device__ __forceinline__ void st32(double *p, const double *v) {  // 4 values
  asm volatile("st.global.cs.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(v[0]), "d"(v[1]), "d"(v[2]), "d"(v[3])
               : "memory");
}
// 8 consecutive values
template <typename T>
__device__ __forceinline__ void ld8_wide(const T *p, T *v) {
  ld32(p, v);
  if constexpr (sizeof(T) == 8) ld32(p + 4, v + 4);
}

}  // namespace mk
