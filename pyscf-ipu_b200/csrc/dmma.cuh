// Float64 matrix instruction m16n8k8 (c += a b).  Lane (g, t) = (lane / 4, lane % 4) holds
// a: rows g, g + 8 at column t, then the same rows at column t + 4; b: rows t, t + 4 of column g;
// c: row g at columns 2 t, 2 t + 1, then row g + 8.
#pragma once
__device__ __forceinline__ void b2_dmma(double (&c)[4], const double (&a)[4], const double (&b)[2]) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
               : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}
