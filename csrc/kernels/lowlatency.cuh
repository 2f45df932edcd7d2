// Lines of the low-latency ("LL") kinds: the flag travels inside the data.
#pragma once
#include "prims.cuh"

namespace fcxdev {

// A 16-byte LL line carries 8 payload bytes and two copies of the 32-bit
// sequence tag: {d0, tag, d1, tag}.  Each 8-byte half is written atomically,
// so a reader that sees the tag in a half also sees that half's payload.
__device__ __forceinline__ void llStore(char *line, uint32_t d0, uint32_t d1, uint32_t tag) {
  asm volatile("st.relaxed.sys.global.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(line), "r"(d0), "r"(tag), "r"(d1), "r"(tag)
               : "memory");
}
__device__ __forceinline__ uint4 llLoad(const char *line) {
  uint4 v;
  asm volatile("ld.relaxed.sys.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(line) : "memory");
  return v;
}

}  // namespace fcxdev
