// Positions on their way between the tiles of the many-step kernels
// (resident.cu, streamed.cu): a double and its step's tag in one 16-byte
// packet.  Each 8-byte half holds half of the double beside the tag, so a
// reader needs no fence and no flag: the packet is complete when both tags
// match.
#pragma once

#include "internal.cuh"

namespace msb {
namespace packets {

__device__ __forceinline__ void put_packet(ulonglong2* p, double v, unsigned tag) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const unsigned long long t = (unsigned long long)tag << 32;
    const unsigned long long lo = (b & 0xffffffffULL) | t, hi = (b >> 32) | t;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(lo), "l"(hi) : "memory");
}

__device__ __forceinline__ void get_packet(const ulonglong2* p, unsigned long long& lo, unsigned long long& hi) {
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(lo), "=l"(hi) : "l"(p) : "memory");
}

__device__ __forceinline__ bool packet_is(unsigned long long lo, unsigned long long hi, unsigned tag) {
    return (unsigned)(lo >> 32) == tag && (unsigned)(hi >> 32) == tag;
}

// Whether a wait that missed its packet for the `spin`-th time (from 0) is over.
// The clock is read, first into t0, from the `patience`-th miss on.
__device__ __forceinline__ bool wait_is_over(int spin, int patience, long long& t0, long long limit) {
    if (spin < patience) return false;
    if (spin == patience) t0 = clock64();
    return clock64() - t0 >= limit;
}

__device__ __forceinline__ double packet_value(unsigned long long lo, unsigned long long hi) {
    return __longlong_as_double((long long)((lo & 0xffffffffULL) | (hi << 32)));
}

}  // namespace packets
}  // namespace msb
