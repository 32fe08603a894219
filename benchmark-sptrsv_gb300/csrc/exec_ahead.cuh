// Polls and publications shared by the executors that stage their lists ahead.
#pragma once
#include "exec_common.cuh"

namespace sptrsv {

// One poll of the R adjacent words of a dependency (pairs by two-word loads): from
// the window in shared memory when `mine`, else from global memory; lanes that do
// not `look` get the empty pattern and load nothing.
__device__ __forceinline__ void poll_words(unsigned long long (&v)[1], unsigned local, const double* word, bool mine,
                                           bool look) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %3, 0;\n\tsetp.ne.u32 q, %4, 0;\n\tmov.u64 %0, -1;\n\t"
      "@p ld.volatile.shared.u64 %0, [%1];\n\t@q ld.relaxed.gpu.global.u64 %0, [%2];\n\t}"
      : "=&l"(v[0])
      : "r"(local), "l"(word), "r"((unsigned)(mine && look)), "r"((unsigned)(!mine && look))
      : "memory");
}
__device__ __forceinline__ void poll_words(unsigned long long (&v)[2], unsigned local, const double* word, bool mine,
                                           bool look) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %4, 0;\n\tsetp.ne.u32 q, %5, 0;\n\tmov.u64 %0, -1;\n\tmov.u64 %1, -1;\n\t"
      "@p ld.volatile.shared.v2.u64 {%0, %1}, [%2];\n\t@q ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%3];\n\t}"
      : "=&l"(v[0]), "=&l"(v[1])
      : "r"(local), "l"(word), "r"((unsigned)(mine && look)), "r"((unsigned)(!mine && look))
      : "memory");
}
__device__ __forceinline__ void poll_words(unsigned (&v)[1], unsigned local, const float* word, bool mine, bool look) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %3, 0;\n\tsetp.ne.u32 q, %4, 0;\n\tmov.u32 %0, -1;\n\t"
      "@p ld.volatile.shared.u32 %0, [%1];\n\t@q ld.relaxed.gpu.global.u32 %0, [%2];\n\t}"
      : "=&r"(v[0])
      : "r"(local), "l"(word), "r"((unsigned)(mine && look)), "r"((unsigned)(!mine && look))
      : "memory");
}
__device__ __forceinline__ void poll_words(unsigned (&v)[2], unsigned local, const float* word, bool mine, bool look) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %4, 0;\n\tsetp.ne.u32 q, %5, 0;\n\tmov.u32 %0, -1;\n\tmov.u32 %1, -1;\n\t"
      "@p ld.volatile.shared.v2.u32 {%0, %1}, [%2];\n\t@q ld.relaxed.gpu.global.v2.u32 {%0, %1}, [%3];\n\t}"
      : "=&r"(v[0]), "=&r"(v[1])
      : "r"(local), "l"(word), "r"((unsigned)(mine && look)), "r"((unsigned)(!mine && look))
      : "memory");
}
__device__ __forceinline__ void publish_words(double* p, const unsigned long long (&v)[1]) {
  st_relaxed_u64(reinterpret_cast<unsigned long long*>(p), v[0]);
}
__device__ __forceinline__ void publish_words(float* p, const unsigned (&v)[1]) {
  st_relaxed_u32(reinterpret_cast<unsigned*>(p), v[0]);
}
__device__ __forceinline__ void publish_words(double* p, const unsigned long long (&v)[2]) {
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(v[0]), "l"(v[1]) : "memory");
}
__device__ __forceinline__ void publish_words(float* p, const unsigned (&v)[2]) {
  asm volatile("st.relaxed.gpu.global.v2.u32 [%0], {%1, %2};" ::"l"(p), "r"(v[0]), "r"(v[1]) : "memory");
}

template <typename B, typename T>
__device__ __forceinline__ void poll_words(B (&v)[4], unsigned local, const T* word, bool mine, bool look) {
  B lo[2], hi[2];
  poll_words(lo, local, word, mine, look);
  poll_words(hi, local + 2u * (unsigned)sizeof(T), word + 2, mine, look);
  v[0] = lo[0];
  v[1] = lo[1];
  v[2] = hi[0];
  v[3] = hi[1];
}
template <typename B, typename T>
__device__ __forceinline__ void publish_words(T* p, const B (&v)[4]) {
  const B lo[2] = {v[0], v[1]}, hi[2] = {v[2], v[3]};
  publish_words(p, lo);
  publish_words(p + 2, hi);
}

}  // namespace sptrsv
