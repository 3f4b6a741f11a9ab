// Shared-memory slots of the solves with pushed values (sptrsv_push.cu,
// batch_cluster.cu).
#pragma once

#include "internal.h"

namespace lace {

// the unsolved mark: all ones, told by the high word
__device__ __forceinline__ unsigned head(float v) { return __float_as_uint(v); }
__device__ __forceinline__ unsigned head(double v) { return (unsigned)__double2hiint(v); }

__device__ __forceinline__ float ld_slot(unsigned a, float) {
  float v;
  asm volatile("ld.volatile.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ double ld_slot(unsigned a, double) {
  double v;
  asm volatile("ld.volatile.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void st_mark(unsigned a, float) {
  asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(a), "r"(0xffffffffu) : "memory");
}
__device__ __forceinline__ void st_mark(unsigned a, double) {
  asm volatile("st.volatile.shared.u64 [%0], %1;" ::"r"(a), "l"(~0ull) : "memory");
}
// A destination (dst: CTA << 24 | byte offset of the slot; -1: none) as an
// address: of this CTA's shared memory, of another's, or none, so that the
// stores on the chain are two predicated instructions and no branch.
struct Slot {
  unsigned a;
  int near, far;
};
__device__ __forceinline__ Slot slot_of(unsigned smem, int rank, int dst) {
  Slot s;
  s.a = smem + (unsigned)(dst & 0xffffff);
  s.near = dst >= 0 && (dst >> 24) == rank;
  s.far = dst >= 0 && !s.near;
  if (s.far) asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(s.a) : "r"(s.a), "r"(dst >> 24));
  return s;
}
__device__ __forceinline__ void push(const Slot &s, float v) {
  asm volatile("{ .reg .pred p, q; setp.ne.s32 p, %1, 0; setp.ne.s32 q, %2, 0; @p st.volatile.shared.f32 [%0], %3; "
               "@q st.relaxed.cluster.shared::cluster.f32 [%0], %3; }" ::"r"(s.a), "r"(s.near), "r"(s.far), "f"(v)
               : "memory");
}
__device__ __forceinline__ void push(const Slot &s, double v) {
  asm volatile("{ .reg .pred p, q; setp.ne.s32 p, %1, 0; setp.ne.s32 q, %2, 0; @p st.volatile.shared.f64 [%0], %3; "
               "@q st.relaxed.cluster.shared::cluster.f64 [%0], %3; }" ::"r"(s.a), "r"(s.near), "r"(s.far), "d"(v)
               : "memory");
}

}  // namespace lace
