// Packed FP32 arithmetic: two products, sums or multiply-adds per instruction,
// each rounded as its scalar form. The rate per value is the scalar one (two
// cycles of the FP32 pipe), but a pair takes one issue slot instead of two,
// which is what bounds the kernels that use it.
//
// A chain of separately rounded products and sums packs one of the two only:
// the compiler fuses a packed product and a packed sum of it into a
// multiply-add, which rounds once.
#pragma once

namespace pikgpu {

// p0 = x0 y0, p1 = x1 y1.
__device__ __forceinline__ void Mul2(float& p0, float& p1, float x0, float x1,
                                     float y0, float y1) {
  asm("{\n\t.reg .b64 x, y;\n\t"
      "mov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
      "mul.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "=f"(p0), "=f"(p1)
      : "f"(x0), "f"(x1), "f"(y0), "f"(y1));
}

// s0 += x0, s1 += x1.
__device__ __forceinline__ void Add2(float& s0, float& s1, float x0,
                                     float x1) {
  asm("{\n\t.reg .b64 s, x;\n\t"
      "mov.b64 s, {%0, %1};\n\tmov.b64 x, {%2, %3};\n\t"
      "add.rn.f32x2 s, s, x;\n\tmov.b64 {%0, %1}, s;\n\t}"
      : "+f"(s0), "+f"(s1)
      : "f"(x0), "f"(x1));
}

// s0 = fmaf(x, y0, s0), s1 = fmaf(x, y1, s1).
__device__ __forceinline__ void Fma2(float& s0, float& s1, float x, float y0,
                                     float y1) {
  asm("{\n\t.reg .b64 s, x, y;\n\t"
      "mov.b64 s, {%0, %1};\n\tmov.b64 x, {%2, %2};\n\t"
      "mov.b64 y, {%3, %4};\n\t"
      "fma.rn.f32x2 s, x, y, s;\n\tmov.b64 {%0, %1}, s;\n\t}"
      : "+f"(s0), "+f"(s1)
      : "f"(x), "f"(y0), "f"(y1));
}

}  // namespace pikgpu
