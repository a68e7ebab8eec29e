// A (value, tag) word moved between blocks as 16 bytes: written and read
// whole, so that a reader that finds the tag it waits for has the value, with
// no fence on either side.
#pragma once

#include <cuda_runtime.h>

namespace pbg {

struct alignas(16) TagWord { unsigned long long v, tag; };

__device__ __forceinline__ TagWord word_ld(const TagWord *p) {
  TagWord w;
  asm volatile("{\n\t.reg .b128 q;\n\tld.relaxed.gpu.global.b128 q, [%2];\n\tmov.b128 {%0, %1}, q;\n\t}"
               : "=l"(w.v), "=l"(w.tag) : "l"(p) : "memory");
  return w;
}
__device__ __forceinline__ void word_st(TagWord *p, double v, unsigned long long tag) {
  asm volatile("{\n\t.reg .b128 q;\n\tmov.b128 q, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], q;\n\t}"
               :: "l"(p), "l"((unsigned long long)__double_as_longlong(v)), "l"(tag) : "memory");
}

}  // namespace pbg
