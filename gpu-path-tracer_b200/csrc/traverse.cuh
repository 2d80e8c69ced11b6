// BVH8 traversal primitives: quantised 8-child box test and the Moller-Trumbore
// triangle test, shared by the closest-hit and any-hit kernels.
#pragma once
#include "pt_internal.h"
#include "pt_math.cuh"

namespace pt
{
    // Per-ray values the node tests need (the direction itself is only needed by triangle tests,
    // which take it separately).
    struct RayPre
    {
        float3 o, invd;
        float tmin;
        uint32_t oct;   // child visiting order: bit k set when the ray's k-th direction component is negative
                        // (near to far); the any-hit kernel flips all three bits (far to near)
    };

    PT_HD float safe_inv(float dk)
    {
        float inv = 1.0f / dk;
        if (!(fabsf(inv) <= 1e30f)) inv = copysignf(1e30f, dk);
        return inv;
    }

    PT_HD RayPre make_ray(float3 o, float3 d, float tmin)
    {
        RayPre r;
        r.o = o;
        r.tmin = tmin;
        r.invd = make_float3(safe_inv(d.x), safe_inv(d.y), safe_inv(d.z));
        r.oct = (r.invd.x < 0.0f ? 1u : 0u) | (r.invd.y < 0.0f ? 2u : 0u) | (r.invd.z < 0.0f ? 4u : 0u);
        return r;
    }

    // Node test. Per child it converts 6 bytes, does 6 multiply-adds, 4 min/max and collects one bit. Byte to
    // float conversions run on the XU pipe (16 a clock per SM), which was the busiest one: 48 of them per visit
    // kept it 62 % busy with 1.5 warps waiting for it per issue. So one axis gets its bytes by a byte permute
    // (ALU pipe) as 1 + q / 32768, the bias folded into the axis' offset. Frame of spheres-1m (1920x1080x64): no
    // axis 92.6 ms, one 90.3, two 91.5, three about 93 (the ALU pipe, which runs the min/max, is then the
    // busier one). Three-input min/max and the sign of (exit - entry) shifted into the mask take 2 fewer ALU
    // operations per child than two-input ones and a compare and select (0.9 ms). Packed f32x2 multiply-adds
    // need their operands in register pairs and were 1 ms slower.
    template <int K>
    __device__ __forceinline__ float byte_of(uint32_t w)
    {
        return static_cast<float>((w >> (8 * K)) & 0xFFu);
    }
    template <int K>
    __device__ __forceinline__ float biased_byte_of(uint32_t w)  // 1 + q / 32768: the byte in the middle of the mantissa
    {
        return __uint_as_float(__byte_perm(w, 0x3F800000u, 0x7604u | (static_cast<uint32_t>(K) << 4)));
    }

    // One axis of a node in ray space: plane q lies at q a + b, with b lowered for near planes and raised for
    // far ones. Rounding of b and of the multiply-add is below 5 ulp of (|b| + 256 |a|), and 2^-20 of it is
    // taken. A biased axis keeps 32768 a in `a` and b - 32768 a in the offsets, whose rounding is at most
    // 2^-9 |a|; 2^-8 |a| is taken. Where 32768 a overflows, the planes become NaN, which the min/max ignore.
    struct SlabAxis
    {
        float a, near, far;
        uint32_t nearLo, nearHi, farLo, farHi;  // bytes of the planes the ray meets first and last, children 0-3 and 4-7
    };

    template <bool BIASED>
    __device__ __forceinline__ SlabAxis slab_axis(float origin, float scale, float invd, uint32_t loLo, uint32_t loHi, uint32_t hiLo, uint32_t hiHi)
    {
        const float kEps = 9.5367431640625e-07f;  // 2^-20
        SlabAxis s;
        s.a = scale * invd;  // (scale: 32768 times the axis' scale when BIASED)
        const float b = origin * invd;
        const float e = __fmaf_rn(BIASED ? 0.125f : 256.0f, fabsf(s.a), fabsf(b));
        s.near = __fmaf_rn(-kEps, e, b);
        s.far = __fmaf_rn(kEps, e, b);
        if constexpr (BIASED)
        {
            s.near = __fsub_rn(s.near, s.a);
            s.far = __fsub_rn(s.far, s.a);
        }
        const bool negative = invd < 0.0f;
        s.nearLo = negative ? hiLo : loLo;
        s.nearHi = negative ? hiHi : loHi;
        s.farLo = negative ? loLo : hiLo;
        s.farHi = negative ? loHi : hiHi;
        return s;
    }

    template <int S, bool BIASED>
    __device__ __forceinline__ float slab_plane(uint32_t lo, uint32_t hi, float a, float b)
    {
        const uint32_t w = S < 4 ? lo : hi;
        if constexpr (BIASED) return __fmaf_rn(biased_byte_of<(S & 3)>(w), a, b);
        else return __fmaf_rn(byte_of<(S & 3)>(w), a, b);
    }

    __device__ __forceinline__ float max3f(float a, float b, float c)
    {
        float r;
        asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
        return r;
    }
    __device__ __forceinline__ float min3f(float a, float b, float c)
    {
        float r;
        asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
        return r;
    }

    // Shifts 1 into `missed` when the ray misses child S, else 0. FIXED (tmin close to 0): the entry distance is
    // clamped to 0 by the three-input integer maximum with a zero floor (the bits of floats that are not negative
    // order like integers; NaNs stay NaNs or are ignored), which takes one operation less than a clamp to tmin.
    template <int S, bool FIXED>
    __device__ __forceinline__ void slab_child(const SlabAxis& x, const SlabAxis& y, const SlabAxis& z, float tmin, float tmax, uint32_t& missed)
    {
        const float nx = slab_plane<S, true>(x.nearLo, x.nearHi, x.a, x.near);
        const float ny = slab_plane<S, false>(y.nearLo, y.nearHi, y.a, y.near);
        const float nz = slab_plane<S, false>(z.nearLo, z.nearHi, z.a, z.near);
        const float fx = slab_plane<S, true>(x.farLo, x.farHi, x.a, x.far);
        const float fy = slab_plane<S, false>(y.farLo, y.farHi, y.a, y.far);
        const float fz = slab_plane<S, false>(z.farLo, z.farHi, z.a, z.far);
        const float tn = FIXED ? __int_as_float(__vimax3_s32_relu(__float_as_int(nx), __float_as_int(ny), __float_as_int(nz)))
                               : fmaxf(max3f(nx, ny, nz), tmin);
        const float tf = fminf(min3f(fx, fy, fz), tmax);
        missed = __funnelshift_l(__float_as_uint(tf - tn), missed, 1);
    }

    // A node's origin relative to the ray's, and its box scales.
    // unit = 2^(u - 127) is 2^-8 of the origin's grid (the low byte of a word is masked, so it holds
    // 256 q); the shift leaves a bit of q in the sign, which fabsf drops. Scales are unit * 2^(e + 1).
    // Powers of two: origin and scale are exact, and d rounds once.
    struct NodeFrame
    {
        float3 d, s;
    };
    __device__ __forceinline__ NodeFrame node_frame(uint4 w0, const RayPre& r)
    {
        const float unit = fabsf(as_float(w0.y << 23));
        NodeFrame f;
        f.s = make_float3(as_float(((w0.z << 23) & 0x0F800000u) | 0x40000000u) * unit, as_float(((w0.w << 23) & 0x0F800000u) | 0x40000000u) * unit,
                          as_float(((w0.z << 18) & 0x03800000u) | ((w0.w << 21) & 0x0C000000u) | 0x40000000u) * unit);
        f.d = make_float3(__fmaf_rn(static_cast<float>(static_cast<int32_t>(w0.x & ~0xFFu)), unit, -r.o.x),
                          __fmaf_rn(static_cast<float>(static_cast<int32_t>(w0.y & ~0xFFu)), unit, -r.o.y),
                          __fmaf_rn(static_cast<float>(static_cast<int32_t>(w0.z & ~0xFFu)), unit, -r.o.z));
        return f;
    }

    // Slab test of the 8 quantised children against [tmin, tmax], conservative for every child box (a box the
    // exact arithmetic would hit is never culled). Returns the hit mask in slot order. Empty slots hold inverted
    // boxes and are almost always culled; one that passes is a record of zeros, which no ray hits.
    template <bool FIXED>
    __device__ __forceinline__ uint32_t intersect_children(uint4 w0, uint4 w1, uint4 w2, uint4 w3, const RayPre& r, float tmin, float tmax)
    {
        const NodeFrame f = node_frame(w0, r);
        // qlo.x = w1.xy, qlo.y = w1.zw, qlo.z = w2.xy, qhi.x = w2.zw, qhi.y = w3.xy, qhi.z = w3.zw
        const SlabAxis x = slab_axis<true>(f.d.x, f.s.x * 32768.0f, r.invd.x, w1.x, w1.y, w2.z, w2.w);
        const SlabAxis y = slab_axis<false>(f.d.y, f.s.y, r.invd.y, w1.z, w1.w, w3.x, w3.y);
        const SlabAxis z = slab_axis<false>(f.d.z, f.s.z, r.invd.z, w2.x, w2.y, w3.z, w3.w);
        uint32_t missed = 0;
        slab_child<7, FIXED>(x, y, z, tmin, tmax, missed);
        slab_child<6, FIXED>(x, y, z, tmin, tmax, missed);
        slab_child<5, FIXED>(x, y, z, tmin, tmax, missed);
        slab_child<4, FIXED>(x, y, z, tmin, tmax, missed);
        slab_child<3, FIXED>(x, y, z, tmin, tmax, missed);
        slab_child<2, FIXED>(x, y, z, tmin, tmax, missed);
        slab_child<1, FIXED>(x, y, z, tmin, tmax, missed);
        slab_child<0, FIXED>(x, y, z, tmin, tmax, missed);
        return ~missed & 0xFFu;
    }

    // The same test for child c alone, with its entry distance.
    __device__ __forceinline__ bool intersect_child(uint4 w0, uint4 w1, uint4 w2, uint4 w3, const RayPre& r, uint32_t c, float tmin, float tmax, float& tn)
    {
        const NodeFrame f = node_frame(w0, r);
        const SlabAxis x = slab_axis<false>(f.d.x, f.s.x, r.invd.x, w1.x, w1.y, w2.z, w2.w);
        const SlabAxis y = slab_axis<false>(f.d.y, f.s.y, r.invd.y, w1.z, w1.w, w3.x, w3.y);
        const SlabAxis z = slab_axis<false>(f.d.z, f.s.z, r.invd.z, w2.x, w2.y, w3.z, w3.w);
        const uint32_t shift = (c & 3u) * 8u;
        const bool high = c >= 4u;
        const auto plane = [&](uint32_t lo, uint32_t hi, float a, float b)
        { return __fmaf_rn(static_cast<float>(((high ? hi : lo) >> shift) & 0xFFu), a, b); };
        tn = fmaxf(max3f(plane(x.nearLo, x.nearHi, x.a, x.near), plane(y.nearLo, y.nearHi, y.a, y.near), plane(z.nearLo, z.nearHi, z.a, z.near)), tmin);
        const float tf = fminf(min3f(plane(x.farLo, x.farHi, x.a, x.far), plane(y.farLo, y.farHi, y.a, y.far), plane(z.farLo, z.farHi, z.a, z.far)), tmax);
        return !(tn > tf);
    }

    // Moller-Trumbore with the reference's determinant cull and inclusive edges
    // (Intersect.cu:25-61), one IEEE rounding per operator. Returns false on a miss;
    // on a barycentric hit returns true with t, u, v (the caller applies the t range).
    PT_HD bool intersect_triangle(float4 a, float4 b, float4 c, float3 o, float3 d, float& t, float& u, float& v)
    {
        const float3 v0 = make_float3(a.x, a.y, a.z);
        const float3 e1 = make_float3(b.x, b.y, b.z);
        const float3 e2 = make_float3(c.x, c.y, c.z);
        const float3 p = mt_cross(d, e2);
        const float det = mt_dot(e1, p);
        if (fabsf(det) < 1e-7f) return false;
        const float3 s = o - v0;
        const float sp = mt_dot_sp(s, p);
        // u = sp * (1/det) is negative when sp and det have opposite signs and the product does not
        // round to zero; with |sp| > 1e-20 and |det| < 1e20 its magnitude exceeds 1e-40, so the
        // reference's u < 0 rejection is decided here without the division (same outcome, bit for bit).
        if (fabsf(sp) > 1e-20f && fabsf(det) < 1e20f && (sp < 0.0f) != (det < 0.0f)) return false;
        const float invDet = 1.0f / det;
        u = sp * invDet;
        if (u < 0.0f || u > 1.0f) return false;
        const float3 q = mt_cross(s, e1);
        v = mt_dot(d, q) * invDet;
        if (v < 0.0f || u + v > 1.0f) return false;
        t = mt_dot(e2, q) * invDet;
        return true;
    }

    struct HitRecord
    {
        float t;
        uint32_t tri;    // input-order triangle index, kInvalid when none
        float u, v;
        uint32_t model;
    };
}
