// Records read and written again by one thread with 256-bit accesses: each read has to see the write before it.
#include "wide_access.cuh"

// before[i], between[i], after[i]: record i (two float4) as read at first, behind a 256-bit write of the record
// plus 1, and behind a plain write of its second half plus 2.
__global__ void rewrite_kernel(float4* records, float4* before, float4* between, float4* after, unsigned n)
{
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4* r = records + 2u * i;
    float4 a, b, c, d, e, f;
    pt::load8(r, a, b);
    pt::store8(r, make_float4(a.x + 1.0f, a.y + 1.0f, a.z + 1.0f, a.w + 1.0f), make_float4(b.x + 1.0f, b.y + 1.0f, b.z + 1.0f, b.w + 1.0f));
    pt::load8(r, c, d);
    r[1] = make_float4(d.x + 2.0f, d.y + 2.0f, d.z + 2.0f, d.w + 2.0f);
    pt::load8(r, e, f);
    before[2u * i] = a;
    before[2u * i + 1u] = b;
    between[2u * i] = c;
    between[2u * i + 1u] = d;
    after[2u * i] = e;
    after[2u * i + 1u] = f;
}

extern "C" int wide_rewrite(float* records, float* before, float* between, float* after, unsigned n, void* stream)
{
    rewrite_kernel<<<(n + 127u) / 128u, 128, 0, static_cast<cudaStream_t>(stream)>>>(
        reinterpret_cast<float4*>(records), reinterpret_cast<float4*>(before), reinterpret_cast<float4*>(between), reinterpret_cast<float4*>(after), n);
    return cudaGetLastError();
}
