// Decoding of the NVFP4 element and scale formats, shared by the projection and quantiser kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace sb {

// E4M3FN decode (nvfp4.c:25-39) for the finite codes.
__device__ __forceinline__ float e4m3_decode(uint32_t code) {
    const uint32_t ex = (code >> 3) & 15u, man = code & 7u;
    float v;
    if (ex == 0) v = __fmul_rn((float)man, 0.001953125f);
    else if (ex == 15 && man == 7) v = __int_as_float(0x7fc00000);
    else v = __uint_as_float(((ex + 120u) << 23) | (man << 20));
    return (code & 0x80u) ? -v : v;
}

// Four E2M1 codes of one half-word as floats, by the hardware conversion (two codes -> f16x2, exact: every E2M1
// value is an f16).  It decodes the code 8 as -0 where the reference's table has +0.
__device__ __forceinline__ void e2m1x4(uint32_t h, float (&f)[4]) {
    uint32_t p0, p1;
    asm("{ .reg .b8 b0, b1;\n\t"
        "mov.b16 {b0, b1}, %2;\n\t"
        "cvt.rn.f16x2.e2m1x2 %0, b0;\n\t"
        "cvt.rn.f16x2.e2m1x2 %1, b1; }\n"
        : "=r"(p0), "=r"(p1)
        : "h"((unsigned short)h));
    asm("{ .reg .b16 l, u;\n\t"
        "mov.b32 {l, u}, %2;\n\t"
        "cvt.f32.f16 %0, l;\n\t"
        "cvt.f32.f16 %1, u; }\n"
        : "=f"(f[0]), "=f"(f[1])
        : "r"(p0));
    asm("{ .reg .b16 l, u;\n\t"
        "mov.b32 {l, u}, %2;\n\t"
        "cvt.f32.f16 %0, l;\n\t"
        "cvt.f32.f16 %1, u; }\n"
        : "=f"(f[2]), "=f"(f[3])
        : "r"(p1));
}

}  // namespace sb
