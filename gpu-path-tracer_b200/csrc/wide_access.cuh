// 256-bit accesses of 32-byte aligned records (sm_100).
#pragma once
#include <cuda_runtime.h>

namespace pt
{
    // 32 read-only bytes in one 256-bit load (sm_100); p must be 32-byte aligned. Halves the load
    // instructions of a node visit and of a triangle test against 16-byte loads.
    __device__ __forceinline__ void ldg8(const uint4* p, uint4& a, uint4& b)
    {
        asm("ld.global.nc.v8.u32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
            : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
            : "l"(p));
    }

    // 32 bytes of memory that kernels write (32-byte aligned). Queue entries are 32-byte records (and 16 bytes more
    // for hits and shadow radiance), which halves the accesses of refilling and retiring rays against arrays of
    // float4: spheres-1m frame (1920x1080x64) closest hits 36.3 -> 35.8 ms, regeneration 4.56 -> 4.46 ms.
    // Volatile and with the memory clobber: a load is not merged with another one or moved over a store (a thread
    // reads a path slot and overwrites it).
    __device__ __forceinline__ void load8(const float4* p, float4& a, float4& b)
    {
        asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
            : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
            : "l"(p)
            : "memory");
    }
    __device__ __forceinline__ void store8(float4* p, float4 a, float4 b)
    {
        asm volatile("st.global.v8.f32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};"
            :: "f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w), "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w), "l"(p) : "memory");
    }
}
