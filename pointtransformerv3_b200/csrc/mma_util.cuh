// Small PTX wrappers shared by the warp-level tensor-core kernels.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

namespace ptv3 {

__device__ __forceinline__ uint32_t smem_u32(const void* p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void cp_async16(uint32_t saddr, const void* gptr)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(saddr), "l"(gptr));
}
// 16-byte copy that writes zeros when `valid` is false (nothing is read then)
__device__ __forceinline__ void cp_async16_zfill(uint32_t saddr, const void* gptr, bool valid)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(saddr), "l"(gptr), "r"(valid ? 16 : 0));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t saddr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(saddr));
}

__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t saddr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(saddr));
}

// D += A(16x16, row) * B(16x8, col), bf16 operands, fp32 accumulate
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi)
{
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

__device__ __forceinline__ float fast_exp2(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
    return y;
}

// two base-2 exponentials of a packed bf16 pair in one instruction
__device__ __forceinline__ uint32_t exp2_bf16x2(uint32_t x)
{
    uint32_t y;
    asm("ex2.approx.ftz.bf16x2 %0, %1;\n" : "=r"(y) : "r"(x));
    return y;
}

// Packed fp32 pairs (two floats in one 64-bit register, one instruction for both).
__device__ __forceinline__ uint64_t pack2(float x, float y)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t r, float& x, float& y)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(r));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b)
{
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b)
{
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// a pair from two 32-bit words (low word = first of the pair)
__device__ __forceinline__ uint64_t pack2u(uint32_t lo, uint32_t hi)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
// a bf16x2 word as a pair of floats
__device__ __forceinline__ uint64_t unpack_bf16x2(uint32_t w) { return pack2u(w << 16, w & 0xffff0000u); }
// both floats rounded to bf16 (round to nearest even); `packed` receives the bf16x2 word
__device__ __forceinline__ uint64_t round2(uint64_t v, uint32_t& packed)
{
    float lo, hi;
    unpack2(v, lo, hi);
    packed = pack_bf16(lo, hi);
    return unpack_bf16x2(packed);
}
__device__ __forceinline__ float hsum2(uint64_t v)
{
    float lo, hi;
    unpack2(v, lo, hi);
    return lo + hi;
}

// acc + the squares of a bf16 pair
__device__ __forceinline__ float sq_norm_bf16x2(uint32_t v, float acc)
{
    const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v));
    return fmaf(f.x, f.x, fmaf(f.y, f.y, acc));
}
// squared norm of 8 bf16 values
__device__ __forceinline__ float sq_norm8(const uint4& a, float acc = 0.f)
{
    return sq_norm_bf16x2(a.x, sq_norm_bf16x2(a.y, sq_norm_bf16x2(a.z, sq_norm_bf16x2(a.w, acc))));
}
// and of 16
__device__ __forceinline__ float sq_norm16(const uint4& a, const uint4& b) { return sq_norm8(b, sq_norm8(a)); }
// maximum that keeps a NaN
__device__ __forceinline__ float max_nan(float a, float b)
{
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

}  // namespace ptv3
