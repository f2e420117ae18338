// ug_dmma.cuh -- FP64 tensor products.
#pragma once

namespace ug {

// D += A B.  8 x 8 x 4: lane (g, t) = (lane / 4, lane % 4) holds A(g, t), B(t, g) and
// D(g, 2t), D(g, 2t + 1).  16 x 8 x 8: A(g, t), A(g + 8, t), A(g, t + 4), A(g + 8, t + 4);
// B(t, g), B(t + 4, g); D(g, 2t), D(g, 2t + 1), D(g + 8, 2t), D(g + 8, 2t + 1).
// Each element accumulates its products in ascending order, one rounding each: the same
// bits as a chain of fused multiply-adds (not promised by PTX; the parity tests pin it).
__device__ __forceinline__ void dmma_8x8x4(double* d, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}
__device__ __forceinline__ void dmma_16x8x8(double* d, const double* a, const double* b) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

}  // namespace ug
