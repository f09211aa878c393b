// f32x2.cuh -- two FP32 operations in one instruction, each rounded as its scalar form.
#pragma once

namespace tam {
namespace {

#define TAM_F32X2(name, op)                                                                                  \
    __device__ __forceinline__ float2 name(float2 a, float2 b)                                               \
    {                                                                                                        \
        float2 r;                                                                                            \
        asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t" op                     \
            ".rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"                                                \
            : "=f"(r.x), "=f"(r.y)                                                                           \
            : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));                                                       \
        return r;                                                                                            \
    }
TAM_F32X2(add2, "add")
TAM_F32X2(sub2, "sub")
TAM_F32X2(mul2, "mul")
#undef TAM_F32X2
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c)
{
    float2 r;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\t"
        "fma.rn.f32x2 x, x, y, z;\n\tmov.b64 {%0, %1}, x;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return r;
}
__device__ __forceinline__ float2 dup(float a) { return make_float2(a, a); }

}  // namespace
}  // namespace tam
