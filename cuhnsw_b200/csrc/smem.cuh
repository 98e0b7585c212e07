// Shared memory by 32-bit address, taken once, instead of generic pointers kept in structs.  Counters of the warp kernel
// (20 000 queries, 1.18 M x 50, ef 200): 374 warp instructions per expansion with pointers, 325 with addresses, conditions
// that are the same in every lane (beam.cuh) and the descent in a kernel of its own (search.cu).
#pragma once
#include <cuda_runtime.h>

namespace hnsw {

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
// an address the compiler keeps in a register instead of deriving it again at each use
__device__ __forceinline__ unsigned kept(unsigned at) {
  unsigned v;
  asm volatile("mov.u32 %0, %1;" : "=r"(v) : "r"(at));
  return v;
}

__device__ __forceinline__ unsigned lds32(unsigned at) {
  unsigned v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(at) : "memory");
  return v;
}
__device__ __forceinline__ uint2 lds64(unsigned at) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(at) : "memory");
  return v;
}
__device__ __forceinline__ uint4 lds128(unsigned at) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at) : "memory");
  return v;
}
__device__ __forceinline__ void sts32(unsigned at, unsigned v) {
  asm volatile("st.shared.u32 [%0], %1;" : : "r"(at), "r"(v) : "memory");
}
__device__ __forceinline__ void sts64(unsigned at, unsigned x, unsigned y) {
  asm volatile("st.shared.v2.u32 [%0], {%1, %2};" : : "r"(at), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void sts128(unsigned at, unsigned x, unsigned y, unsigned z, unsigned w) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" : : "r"(at), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ unsigned atomic_add_shared(unsigned at, unsigned v) {
  unsigned old;
  asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(at), "r"(v) : "memory");
  return old;
}

__device__ __forceinline__ void atomic_or_shared(unsigned at, unsigned v) {
  asm volatile("red.shared.or.b32 [%0], %1;" : : "r"(at), "r"(v) : "memory");
}

__device__ __forceinline__ void atomic_min_shared(unsigned at, unsigned v) {
  asm volatile("red.shared.min.u32 [%0], %1;" : : "r"(at), "r"(v) : "memory");
}

// where `on`, the cache line of global memory at p on its way to the L2 cache
__device__ __forceinline__ void prefetch_l2_if(bool on, const void* p) {
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %1, 0;\n @p prefetch.global.L2 [%0];\n}" : : "l"(p), "r"((unsigned)on));
}

// The lane number, read once: the compiler does not fetch it again where registers are short.
__device__ __forceinline__ int lane_number() {
  unsigned v;
  asm volatile("mov.u32 %0, %%laneid;" : "=r"(v));
  return (int)v;
}

}  // namespace hnsw
