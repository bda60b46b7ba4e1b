// Device pieces that the product kernels share: streaming loads of an 8-element unit, the mask of a unit that straddles the
// end of a row, address arithmetic on byte prefix sums and the fp16 multiply-adds.
#pragma once

#include <cuda_fp16.h>

namespace macko {
namespace {

constexpr int kGroup = 8;            // stored elements per lane per sub-step (one 128-bit value load)

template <int V> struct Int { static constexpr int value = V; };

// acc += fp16(half VH of vword) * fp16(half XH of xword)
template <int VH, int XH>
__device__ __forceinline__ float fma_hh(float acc, unsigned vword, unsigned xword)
{
    if (VH == 0 && XH == 0)
        asm("{.reg .b16 vl,vh,xl,xh; mov.b32 {vl,vh}, %1; mov.b32 {xl,xh}, %2; fma.rn.f32.f16 %0, vl, xl, %0;}" : "+f"(acc) : "r"(vword), "r"(xword));
    else if (VH == 0 && XH == 1)
        asm("{.reg .b16 vl,vh,xl,xh; mov.b32 {vl,vh}, %1; mov.b32 {xl,xh}, %2; fma.rn.f32.f16 %0, vl, xh, %0;}" : "+f"(acc) : "r"(vword), "r"(xword));
    else if (VH == 1 && XH == 0)
        asm("{.reg .b16 vl,vh,xl,xh; mov.b32 {vl,vh}, %1; mov.b32 {xl,xh}, %2; fma.rn.f32.f16 %0, vh, xl, %0;}" : "+f"(acc) : "r"(vword), "r"(xword));
    else
        asm("{.reg .b16 vl,vh,xl,xh; mov.b32 {vl,vh}, %1; mov.b32 {xl,xh}, %2; fma.rn.f32.f16 %0, vh, xh, %0;}" : "+f"(acc) : "r"(vword), "r"(xword));
    return acc;
}

// BV consecutive fp16 values (BV = 2, 4 or 8) from shared memory into BV/2 words
template <int BV>
__device__ __forceinline__ void lds_vec(unsigned addr, unsigned (&r)[BV / 2])
{
    if constexpr (BV == 2)
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(r[0]) : "r"(addr));
    else if constexpr (BV == 4)
        asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(addr));
    else
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}

__device__ __forceinline__ uint4 ldg_stream_v4(const uint4 *p)
{
    uint4 r;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
    return r;
}

__device__ __forceinline__ unsigned ldg_stream_u32(const unsigned *p)
{
    unsigned r;
    asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(r) : "l"(p));
    return r;
}

// Loads of what the kernel in front in the stream may have written while this one was already resident (programmatic dependent
// launch): not the read-only path (ld.global.nc, which __ldg and const __restrict__ pointers become), whose data must not change
// while a kernel lives, and volatile, so that they stay behind griddepcontrol.wait.
__device__ __forceinline__ unsigned short ldg_fresh_u16(const void *p)
{
    unsigned short r;
    asm volatile("ld.global.u16 %0, [%1];" : "=h"(r) : "l"(p));
    return r;
}

__device__ __forceinline__ uint2 ldg_fresh_v2(const uint2 *p)
{
    uint2 r;
    asm volatile("ld.global.v2.u32 {%0,%1}, [%2];" : "=r"(r.x), "=r"(r.y) : "l"(p));
    return r;
}

// c + byte `J` of a: one integer dot-product instruction extracts the byte and adds the base, and it
// does not run on the (half-rate) integer ALU pipe the rest of the index arithmetic competes for.
template <int J, int M = 1>
__device__ __forceinline__ int add_byte(unsigned a, int c)
{
    return __dp4a(a, (unsigned)M << (8 * J), (unsigned)c);   // c + M * byte J of a
}

// Zero the deltas and the fp16 values of one 8-element unit outside element range [lo, hi).
__device__ __forceinline__ void mask_unit(uint4 &v, unsigned &w, int lo, int hi)
{
    lo = min(max(lo, 0), kGroup);
    hi = min(max(hi, 0), kGroup);
    unsigned m = lo >= kGroup ? 0u : (0xffffffffu << (4 * lo));
    if (hi < kGroup) m &= ~(0xffffffffu << (4 * hi));
    w &= m;
    unsigned *vw = reinterpret_cast<unsigned *>(&v);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const unsigned lo16 = ((m >> (8 * j)) & 1u) * 0xffffu;
        const unsigned hi16 = ((m >> (8 * j + 4)) & 1u) * 0xffff0000u;
        vw[j] &= (lo16 | hi16);
    }
}

}  // namespace
}  // namespace macko
