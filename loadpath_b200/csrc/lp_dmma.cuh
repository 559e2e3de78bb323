// FP64 tensor-core MMA, m8n8k4 (row-major A 8 x 4, column-major B 4 x 8, C/D 8 x 8). Lane l holds
// A[l >> 2][l & 3], B[l & 3][l >> 2] and D[l >> 2][2 (l & 3) + i], i = 0, 1.
#pragma once

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}
