// Device parts of the MPO stage out[x, q, y] = sum_p M[q, p] in[x, p, y], for CTAs that
// each own one (x, STAGE_Y-wide y chunk): thread q compacts the nonzeros of row q of M in shared memory, the P input rows of the chunk are staged there
// too.
// Bound: HBM / L2 for large tensors, latency for small ones, and close behind both the
// FP64 units (two operations per SM and cycle), so entries are applied by kind: an MPO
// entry is real nearly always (two operations instead of four), often exactly 1 (one
// addition), and the first entry of a row starts the sum instead of being added to zero.
// Measured (separate stage kernel) at bonds 512 x 512, chi 5: 65 -> 37 us; at bonds <= 28:
// 15.9 -> 6.3 us (one thread scanned W before, and every entry took four FMAs).
#pragma once

#include "ptn_common.cuh"

namespace ptn {

constexpr int STAGE_Y = 128;     // columns of a CTA, at least as many threads
constexpr int STAGE_MAX = 64;    // largest P and Q

enum { ENTRY_COMPLEX = 0, ENTRY_REAL = 1, ENTRY_ONE = 2 };

// dynamic shared memory: input rows, row-wise nonzeros and their indices
inline size_t stage_smem(int P, int Q) {
  return (size_t)P * STAGE_Y * sizeof(double2) + (size_t)P * Q * (sizeof(double2) + sizeof(int));
}

// FP64 operations the compiler may not hoist out of their branch: computed for every entry
// whatever its kind, they would cost 64 cycles of a sub-partition each
__device__ __forceinline__ double mul_here(double a, double b) {
  double r;
  asm volatile("mul.rn.f64 %0, %1, %2;" : "=d"(r) : "d"(a), "d"(b));
  return r;
}
__device__ __forceinline__ double fma_here(double a, double b, double c) {
  double r;
  asm volatile("fma.rn.f64 %0, %1, %2, %3;" : "=d"(r) : "d"(a), "d"(b), "d"(c));
  return r;
}
__device__ __forceinline__ double add_here(double a, double b) {
  double r;
  asm volatile("add.rn.f64 %0, %1, %2;" : "=d"(r) : "d"(a), "d"(b));
  return r;
}

static __device__ __noinline__ double2 entry_complex(double2 v, double2 x, double2 acc, int first) {
  return first ? cmul(v, x) : cfma(v, x, acc);
}

__device__ __forceinline__ double2 entry_mul(int kind, double2 v, double2 x) {
  if (kind == ENTRY_ONE) return x;
  if (kind == ENTRY_REAL) return make_double2(mul_here(v.x, x.x), mul_here(v.x, x.y));
  return entry_complex(v, x, x, 1);
}

__device__ __forceinline__ double2 entry_fma(int kind, double2 v, double2 x, double2 acc) {
  if (kind == ENTRY_ONE) return make_double2(add_here(acc.x, x.x), add_here(acc.y, x.y));
  if (kind == ENTRY_REAL)
    return make_double2(fma_here(v.x, x.x, acc.x), fma_here(v.x, x.y, acc.y));
  return entry_complex(v, x, acc, 0);
}

// M (given by strides into w) -> sval[q * P + p]
__device__ __forceinline__ void stage_load_w(const double2* __restrict__ w, long ldq, long ldp,
                                             int P, int Q, double2* sval) {
  for (int e = threadIdx.x; e < P * Q; e += blockDim.x) sval[e] = w[(e / P) * ldq + (e % P) * ldp];
}

// row q of sval -> its nonzeros, their indices 4 * p + kind, their number
__device__ __forceinline__ void stage_compact(int P, int Q, double2* sval, int* sidx, int* scount) {
  const int q = threadIdx.x;
  if (q >= Q) return;
  double2* row = sval + q * P;
  int* idx = sidx + q * P;
  int nz = 0;
  for (int p = 0; p < P; ++p) {
    const double2 v = row[p];
    if (v.x != 0.0 || v.y != 0.0) {
      row[nz] = v;
      idx[nz] = 4 * p + (v.y != 0.0 ? ENTRY_COMPLEX : v.x != 1.0 ? ENTRY_REAL : ENTRY_ONE);
      ++nz;
    }
  }
  scount[q] = nz;
}

// output row q at this thread's column (col: its entry of input row 0)
__device__ __forceinline__ double2 stage_row(int q, int P, const double2* col, const double2* sval,
                                             const int* sidx, const int* scount) {
  const double2* row = sval + q * P;
  const int* idx = sidx + q * P;
  const int nz = scount[q];
  double2 acc = make_double2(0.0, 0.0);
  if (nz > 0) acc = entry_mul(idx[0] & 3, row[0], col[(idx[0] >> 2) * STAGE_Y]);
  for (int e = 1; e < nz; ++e)
    acc = entry_fma(idx[e] & 3, row[e], col[(idx[e] >> 2) * STAGE_Y], acc);
  return acc;
}

}  // namespace ptn
