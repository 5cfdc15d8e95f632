// dmma.cuh -- the FP64 tensor-core instruction of sm_90 and later.
#pragma once

namespace dvr3d {

// One m16n8k16 product, C += A B. With g = lane / 4 and t = lane % 4 the fragments are
// A(g + 8 (i % 2), t + 4 (i / 2)) for a[0..7], B(k = t + 4 i, n = g) for b[0..3], and C(g, 2t),
// C(g, 2t+1), C(g+8, 2t), C(g+8, 2t+1) for c[0..3].
__device__ __forceinline__ void dmma16(double (&c)[4], const double (&a)[8], const double (&b)[4]) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7,%8,%9,%10,%11}, "
        "{%12,%13,%14,%15}, {%0,%1,%2,%3};\n"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]), "d"(a[6]), "d"(a[7]), "d"(b[0]),
          "d"(b[1]), "d"(b[2]), "d"(b[3]));
}

}  // namespace dvr3d
