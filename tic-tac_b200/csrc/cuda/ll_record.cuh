// Records that pass an element of a vector or row between the CTAs of one launch:
// the element and a tag, stored in one 16-byte access that is single-copy atomic
// (complex128: two), so a reader that sees its tag sees the element, without a
// fence or a flag beside the data.
#pragma once
#include <cuda_runtime.h>

namespace tt {

__device__ __forceinline__ void ll_store(void* p, unsigned long long lo, unsigned long long hi) {
  asm volatile("{\n\t.reg .b128 q;\n\tmov.b128 q, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], q;\n\t}" ::"l"(p),
               "l"(lo), "l"(hi)
               : "memory");
}
__device__ __forceinline__ void ll_load(const void* p, unsigned long long& lo, unsigned long long& hi) {
  asm volatile("{\n\t.reg .b128 q;\n\tld.relaxed.gpu.global.b128 q, [%2];\n\tmov.b128 {%0, %1}, q;\n\t}"
               : "=l"(lo), "=l"(hi)
               : "l"(p)
               : "memory");
}
// Programmatic dependent launch.  The kernels of a panel follow one another every few
// microseconds: each lets the next one be launched while it runs, and a kernel launched
// so waits, before its first access to memory, until everything before it in the
// stream is complete; only then does it let its own successor in.  Solves of order
// 1,859 9.25 -> 8.63 ms, 512 1.63 -> 1.55 ms, the adjoint of 10,944 46.6 -> 45.1 ms.
__device__ __forceinline__ void pdl_launch_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// one element of a posted row: complex64 in one record, complex128 in two
template <typename T>
struct LL;
template <>
struct LL<float2> {
  static constexpr int BYTES = 16;
  static __device__ __forceinline__ void post(unsigned char* p, float2 v, unsigned long long hi) {
    ll_store(p, (unsigned long long)__float_as_uint(v.x) | ((unsigned long long)__float_as_uint(v.y) << 32), hi);
  }
  static __device__ __forceinline__ bool poll(const unsigned char* p, float2& v, unsigned long long& hi,
                                              unsigned tag) {
    unsigned long long lo;
    ll_load(p, lo, hi);
    v = make_float2(__uint_as_float((unsigned)lo), __uint_as_float((unsigned)(lo >> 32)));
    return (unsigned)hi == tag;
  }
};
template <>
struct LL<double2> {
  static constexpr int BYTES = 32;
  static __device__ __forceinline__ void post(unsigned char* p, double2 v, unsigned long long hi) {
    ll_store(p, (unsigned long long)__double_as_longlong(v.x), hi);
    ll_store(p + 16, (unsigned long long)__double_as_longlong(v.y), hi);
  }
  static __device__ __forceinline__ bool poll(const unsigned char* p, double2& v, unsigned long long& hi,
                                              unsigned tag) {
    unsigned long long lx, ly, h2;
    ll_load(p, lx, hi);
    ll_load(p + 16, ly, h2);
    v = make_double2(__longlong_as_double((long long)lx), __longlong_as_double((long long)ly));
    return (unsigned)hi == tag && (unsigned)h2 == tag;
  }
};

}  // namespace tt
