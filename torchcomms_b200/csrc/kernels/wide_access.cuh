// 32 bytes of global memory in one access; the address on a 32-byte boundary. Lanes that each take 32 neighbouring bytes in
// two accesses of 16 touch every sector twice.
#pragma once

#include <cuda_runtime.h>

namespace b200c {

#ifdef __CUDACC__

__device__ __forceinline__ void ld32(const void* p, uint4& lo, uint4& hi) {
  asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(lo.x), "=r"(lo.y), "=r"(lo.z), "=r"(lo.w), "=r"(hi.x), "=r"(hi.y), "=r"(hi.z), "=r"(hi.w)
               : "l"(p)
               : "memory");
}
// What is read once.
__device__ __forceinline__ void ld32_stream(const void* p, uint4& lo, uint4& hi) {
  asm volatile("ld.global.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(lo.x), "=r"(lo.y), "=r"(lo.z), "=r"(lo.w), "=r"(hi.x), "=r"(hi.y), "=r"(hi.z), "=r"(hi.w)
               : "l"(p));
}
__device__ __forceinline__ void st32(void* p, uint4 lo, uint4 hi) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(lo.x), "r"(lo.y), "r"(lo.z), "r"(lo.w), "r"(hi.x), "r"(hi.y),
               "r"(hi.z), "r"(hi.w)
               : "memory");
}

#endif // __CUDACC__

} // namespace b200c
