// Asynchronous copies to shared memory, packet by packet, for the streaming block kernels.
#pragma once

namespace momed {

// Asynchronous copies of a thread's own packets to its own places of a ring in shared memory: no other
// thread reads them, so a thread waits for its own copies only.
template <typename PT> __device__ __forceinline__ void copy_packet(PT* dst, const PT* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if constexpr (sizeof(PT) == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

}  // namespace momed
