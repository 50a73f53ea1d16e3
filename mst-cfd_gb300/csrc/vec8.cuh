// 32-byte (one sector) loads and stores of eight floats; the address is
// 32-byte aligned.  One request per record instead of two of 16 bytes.
// (volatile: the load stays behind chain(), see chained.cuh)
#pragma once

namespace mst {

__device__ __forceinline__ void load8(const float* p, float x[8]) {
  asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]), "=f"(x[4]), "=f"(x[5]), "=f"(x[6]),
        "=f"(x[7])
      : "l"(p));
}
__device__ __forceinline__ void store8(float* p, const float x[8]) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(x[0]),
               "f"(x[1]), "f"(x[2]), "f"(x[3]), "f"(x[4]), "f"(x[5]), "f"(x[6]), "f"(x[7])
               : "memory");
}

}  // namespace mst
