// The digit GEMM's entry (ptn_zgemm_split_bf16), which absorbs the bond matrix into the next
// site in the mixed form: conversion of both operands to BF16 digits, exact digit products
// on the tensor cores (tc_gemm.cu). The contractions of the mixed form run in the residue
// number system (rns_ops.cu); this product acts on the state itself once per site, so its
// results stay the ones it always gave, bit for bit.
//
// Operand conversion ("digits"): a complex matrix view (element (r, k) at
// src[r * sr + k * sk]) becomes five BF16 digit planes plus one power-of-two
// exponent per row r. Two tiled passes: the first finds each row's largest
// |component| (atomicMax of the IEEE exponent field), the second forms the
// fixed-point integer round(x 2^(39 - e)) from the IEEE fields and cuts it into
// five balanced base-256 digits with integer arithmetic only, stored k-contiguously. "Plain" operands keep
// re/im interleaved along K; "embedded" operands store z as [[Re, -Im], [Im, Re]].
#include "ptn_common.cuh"
#include <cuda_bf16.h>
#include <algorithm>

namespace ptn {

void note_launches(int n);
ptn_status tc_gemm(const void* Aslices, long aplane, const int* ea, const void* Bslices, long bplane,
                   const int* eb, int M, int Nc, int Kc, long Kp, double2* out, long ldm, long ldn,
                   bool accumulate, void* ws, size_t ws_bytes, const int* skip, cudaStream_t st,
                   const unsigned char* fa, const unsigned char* fb, int fk);
size_t tc_gemm_workspace_bytes(int M, int Ncomplex, int Kcomplex);

namespace {

typedef __nv_bfloat16 bf16;
constexpr int NDIGIT = 5;
constexpr int EXP_ZERO = -2000;   // rows with no non-zero entry (memset 0x80 gives less)

// 32 x 32 complex tile of the view, rows r0.., cols k0..; threads (32, 8)
__device__ __forceinline__ void load_tile(double2 (*tile)[33], const double2* __restrict__ src,
                                          long sr, long sk, int R, int K, int r0, int k0, int conj) {
  const int tx = threadIdx.x, ty = threadIdx.y;
  if (sk == 1) {
    for (int rr = ty; rr < 32; rr += 8) {
      const int r = r0 + rr, k = k0 + tx;
      double2 v = (r < R && k < K) ? src[(long)r * sr + k] : make_double2(0.0, 0.0);
      if (conj) v.y = -v.y;
      tile[rr][tx] = v;
    }
  } else {
    for (int kk = ty; kk < 32; kk += 8) {
      const int r = r0 + tx, k = k0 + kk;
      double2 v = (r < R && k < K) ? src[(long)r * sr + (long)k * sk] : make_double2(0.0, 0.0);
      if (conj) v.y = -v.y;
      tile[tx][kk] = v;
    }
  }
}

__device__ __forceinline__ int biased_exp(double x) {
  return (int)((__double_as_longlong(x) >> 52) & 0x7FF);
}

__global__ void rowexp_kernel(const double2* __restrict__ src, long sr, long sk, int R, int K,
                              int* __restrict__ e, const int* skip) {
  if (skip != nullptr && *skip != 0) return;
  __shared__ double2 tile[32][33];
  const int r0 = blockIdx.y * 32, k0 = blockIdx.x * 32;
  load_tile(tile, src, sr, sk, R, K, r0, k0, 0);
  __syncthreads();
  for (int rr = threadIdx.y; rr < 32; rr += 8) {
    const double2 v = tile[rr][threadIdx.x];
    // biased exponent fields (integer work only; zero and subnormal entries give 0)
    int m = max(biased_exp(v.x), biased_exp(v.y));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (threadIdx.x == 0 && r0 + rr < R && m > 0) {
      // a normal |x| with biased exponent E lies in [2^(E-1023), 2^(E-1022)): every
      // entry of the row is below 2^ex (frexp's exponent of the largest one)
      atomicMax(&e[r0 + rr], m - 1022);
    }
  }
}

// Balanced base-256 digits of x 2^(7 - ex) (|x| < 2^ex): the fixed-point integer
// T = round(x 2^(39 - ex)) (|T| <= 2^39) is cut into
// T = d0 2^32 + d1 2^24 + d2 2^16 + d3 2^8 + d4 with d1..d4 in [-128, 127] and
// |d0| <= 128, each exact in BF16. Integer
// arithmetic on the IEEE fields only: the CUDA-core FP64 rate of this part is low.
// Zero and subnormal entries (below 2^-1022) give zero digits.
__device__ __forceinline__ void digits_of(double x, int ex, bf16 (&d)[NDIGIT]) {
  const long long b = __double_as_longlong(x);
  const int E = (int)((b >> 52) & 0x7FF);
  long long T = 0;
  if (E != 0) {
    const long long mant = (b & ((1LL << 52) - 1)) | (1LL << 52);
    // x = mant 2^(E - 1075): T = round(mant 2^(E - 1075 + 39 - ex)), shift always right
    const int rs = 1075 - (8 * NDIGIT - 1) + ex - E;
    if (rs < 63) T = (rs <= 0) ? (mant << (-rs)) : ((mant + (1LL << (rs - 1))) >> rs);
    if (b < 0) T = -T;
  }
#pragma unroll
  for (int i = NDIGIT - 1; i > 0; --i) {
    const int di = (int)((T + 128) & 255) - 128;
    d[i] = __int2bfloat16_rn(di);
    T = (T - di) >> 8;   // exact
  }
  d[0] = __int2bfloat16_rn((int)T);
}

// With zero-tile flags on (flags_on), also marks flags[1 + (r / fg) * fk + k / 16]
// for every non-zero entry (r, k): the tiles of the digit GEMM (128 rows of a plain
// operand, 48 complex columns of an embedded one) by K block of 16 complex entries,
// so that the GEMM can skip all-zero tiles (quantum-number block sparsity); one
// store per warp, row and K block (the buffer is zeroed before). flags[0] tells the
// GEMM whether the flags of this conversion are valid.
__global__ void digits_kernel(const double2* __restrict__ src, long sr, long sk, int R, int K,
                              int conj, const int* __restrict__ e, bf16* __restrict__ dst, long Kp,
                              long plane, int embedded, unsigned char* __restrict__ flags,
                              int flags_on, int fg, long fk, const int* skip) {
  if (skip != nullptr && *skip != 0) return;
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && threadIdx.y == 0)
    flags[0] = (unsigned char)flags_on;
  __shared__ double2 tile[32][33];
  const int r0 = blockIdx.y * 32, k0 = blockIdx.x * 32;
  load_tile(tile, src, sr, sk, R, K, r0, k0, conj);
  __syncthreads();
  if (flags_on) {
    // lanes 0..15 and 16..31 of a row cover one K block each
    for (int rr = threadIdx.y; rr < 32; rr += 8) {
      const int r = r0 + rr, k = k0 + threadIdx.x;
      const double2 z = tile[rr][threadIdx.x];
      const unsigned nz = __ballot_sync(0xffffffffu, r < R && k < K && (z.x != 0.0 || z.y != 0.0));
      const unsigned half = (threadIdx.x < 16) ? (nz & 0xFFFFu) : (nz >> 16);
      if ((threadIdx.x & 15) == 0 && half != 0) flags[1 + (long)(r / fg) * fk + (k >> 4)] = 1;
    }
  }
  const int k = k0 + threadIdx.x;
  if (k >= K) return;
  for (int rr = threadIdx.y; rr < 32; rr += 8) {
    const int r = r0 + rr;
    if (r >= R) break;
    const int ex = e[r];
    const double2 z = tile[rr][threadIdx.x];
    bf16 dr[NDIGIT], di[NDIGIT];
    if (ex > EXP_ZERO) {
      digits_of(z.x, ex, dr);
      digits_of(z.y, ex, di);
    } else {
#pragma unroll
      for (int i = 0; i < NDIGIT; ++i) dr[i] = di[i] = __double2bfloat16(0.0);
    }
#pragma unroll
    for (int i = 0; i < NDIGIT; ++i) {
      bf16* base = dst + (long)i * plane;
      if (!embedded) {
        reinterpret_cast<__nv_bfloat162*>(base + (long)r * Kp + 2L * k)[0] =
            __halves2bfloat162(dr[i], di[i]);
      } else {
        reinterpret_cast<__nv_bfloat162*>(base + (2L * r) * Kp + 2L * k)[0] =
            __halves2bfloat162(dr[i], __hneg(di[i]));
        reinterpret_cast<__nv_bfloat162*>(base + (2L * r + 1) * Kp + 2L * k)[0] =
            __halves2bfloat162(di[i], dr[i]);
      }
    }
  }
}

inline long kpad(long kc) { return (2 * kc + 63) / 64 * 64; }
inline size_t al(size_t b) { return (b + 255) & ~size_t(255); }

// bump allocator over the caller's workspace (null base: size query)
struct Carver {
  char* base;
  size_t off = 0;
  explicit Carver(void* b) : base(static_cast<char*>(b)) {}
  void* take(size_t bytes) {
    void* p = base ? base + off : nullptr;
    off += al(bytes);
    return p;
  }
};

// BF16 digit planes of a complex matrix with `rows` rows (2 * rows real rows when
// embedded) and kc complex columns, plus the per-row exponents
struct Digits {
  bf16* p;
  int* e;
  unsigned char* f;   // non-zero flags per (GEMM tile of rows, K block of 16 complex)
  long rows, kc, Kp;
  bool embedded;
  int fgroup() const { return embedded ? 48 : 128; }
  long fk() const { return (kc + 15) / 16; }
  long frows() const { return (rows + fgroup() - 1) / fgroup(); }
  long real_rows() const { return embedded ? 2 * rows : rows; }
  long plane() const { return real_rows() * Kp; }
};

Digits take_digits(Carver& c, long rows, long kc, bool embedded) {
  Digits d;
  d.rows = rows;
  d.kc = kc;
  d.Kp = kpad(kc);
  d.embedded = embedded;
  d.p = static_cast<bf16*>(c.take((size_t)NDIGIT * d.real_rows() * d.Kp * sizeof(bf16)));
  d.e = static_cast<int*>(c.take((size_t)rows * sizeof(int)));
  d.f = static_cast<unsigned char*>(c.take(1 + (size_t)d.frows() * d.fk()));
  return d;
}

// view (r, k) -> src[r * sr + k * sk], r < d.rows, k < d.kc
ptn_status to_digits(const double2* src, long sr, long sk, const Digits& d, bool conj,
                     const int* skip, cudaStream_t st) {
  PTN_CUDA_TRY(cudaMemsetAsync(d.e, 0x80, (size_t)d.rows * sizeof(int), st));
  const int flags_on = tune(PTN_TUNE_TC_SKIP_ZERO) != 0 ? 1 : 0;
  if (flags_on) PTN_CUDA_TRY(cudaMemsetAsync(d.f, 0, 1 + (size_t)d.frows() * d.fk(), st));
  dim3 grid((unsigned)((d.kc + 31) / 32), (unsigned)((d.rows + 31) / 32));
  PTN_CHECK_ARG(grid.y <= 65535, "digits: too many rows");
  rowexp_kernel<<<grid, dim3(32, 8), 0, st>>>(src, sr, sk, (int)d.rows, (int)d.kc, d.e, skip);
  digits_kernel<<<grid, dim3(32, 8), 0, st>>>(src, sr, sk, (int)d.rows, (int)d.kc, conj ? 1 : 0,
                                              d.e, d.p, d.Kp, d.plane(), d.embedded ? 1 : 0, d.f,
                                              flags_on, d.fgroup(), d.fk(), skip);
  PTN_LAUNCH_CHECK();
  note_launches(2);
  return PTN_OK;
}

// C = A . B^T over the digit planes: A plain (M x Kc), B embedded (Nc x Kc)
ptn_status gemm(const Digits& A, const Digits& Be, double2* out, long ldm, long ldn, void* ws,
                size_t ws_bytes, const int* skip, cudaStream_t st) {
  const bool flags = tune(PTN_TUNE_TC_SKIP_ZERO) != 0;
  return tc_gemm(A.p, A.plane(), A.e, Be.p, Be.plane(), Be.e, (int)A.rows, (int)Be.rows,
                 (int)A.kc, A.Kp, out, ldm, ldn, false, ws, ws_bytes, skip, st,
                 flags ? A.f : nullptr, flags ? Be.f : nullptr, (int)A.fk());
}

}  // namespace

// ================================================================ plain GEMM entry
size_t zgemm_split_workspace_bytes(int M, int N, int K) {
  Carver c(nullptr);
  take_digits(c, M, K, false);
  take_digits(c, N, K, true);
  c.take(tc_gemm_workspace_bytes(M, N, K));
  return c.off;
}

// C = A B (row-major complex, M x K times K x N) through the digit products
ptn_status zgemm_split(const double2* A, long lda, const double2* B, long ldb, double2* C, long ldc,
                       int M, int N, int K, void* ws, size_t ws_bytes, cudaStream_t st) {
  PTN_CHECK_ARG(M > 0 && N > 0 && K > 0, "zgemm_split: bad sizes");
  Carver c(ws);
  Digits As = take_digits(c, M, K, false);
  Digits Bs = take_digits(c, N, K, true);
  PTN_CHECK_ARG(ws_bytes >= c.off, "zgemm_split: workspace too small");
  void* g = c.take(0);
  const size_t gb = ws_bytes - c.off;
  PTN_TRY(to_digits(A, lda, 1, As, false, nullptr, st));
  // B as the view (n, k) = B[k][n]
  PTN_TRY(to_digits(B, 1, ldb, Bs, false, nullptr, st));
  return gemm(As, Bs, C, ldc, 1, g, gb, nullptr, st);
}

}  // namespace ptn

extern "C" {

size_t ptn_zgemm_split_bf16_workspace_bytes(int M, int N, int K) {
  return ptn::zgemm_split_workspace_bytes(M, N, K);
}

ptn_status ptn_zgemm_split_bf16(const ptn_c128* A, long lda, const ptn_c128* B, long ldb,
                                ptn_c128* C, long ldc, int M, int N, int K, void* ws,
                                size_t ws_bytes, void* stream) {
  return ptn::zgemm_split(reinterpret_cast<const double2*>(A), lda,
                          reinterpret_cast<const double2*>(B), ldb, reinterpret_cast<double2*>(C),
                          ldc, M, N, K, ws, ws_bytes, ptn::as_stream(stream));
}

}  // extern "C"
