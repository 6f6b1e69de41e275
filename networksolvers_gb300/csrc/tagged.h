// Messages between the CTAs of one launch through L2: a double and a tag in one 16-byte access,
// so that a consumer polls the value itself (no counter, no fence, no second round trip).
#pragma once

namespace nsg {

__device__ __forceinline__ void put_tagged(ulonglong2* p, double v, unsigned long long tag) {
  asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}\n" ::"l"(p),
               "l"(__double_as_longlong(v)), "l"(tag)
               : "memory");
}
__device__ __forceinline__ bool get_tagged(const ulonglong2* p, unsigned long long tag, double& v) {
  unsigned long long a, b;
  asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}\n"
               : "=l"(a), "=l"(b)
               : "l"(p)
               : "memory");
  v = __longlong_as_double((long long)a);
  return b == tag;
}

}  // namespace nsg
