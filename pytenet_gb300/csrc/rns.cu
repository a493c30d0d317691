// Complex GEMM in a residue number system on the 5th-generation tensor cores (tcgen05).
//
// C = A B over complex FP64 is computed exactly in integers and rounded once:
//   - every row of A and every column of B is scaled by its own power of two and rounded
//     to Gaussian integers of `bits` bits (53 or 54 in the FP64 form, 39 and more in the
//     mixed form); in the FP64 form the terms are scaled before by powers of two that cancel
//     in the product (RnsTerms in rns.cuh), so that operands which grow and decay against
//     each other along the terms lose nothing;
//   - the integer product is formed modulo nm small pairwise coprime numbers p and put
//     together by the Chinese remainder theorem (Ozaki, Uchino and Imamura, "Ozaki Scheme
//     II", 2025, use it for real matrices). All prime factors of the moduli are 1 mod 4,
//     so -1 has a square root j modulo p and the Gaussian integers modulo p split into two
//     independent copies of the integers modulo p: z = x + i y -> (x + j y, x - j y). A
//     complex product therefore costs two real ones per modulus (not four), conjugation
//     swaps the copies, and the copies of all moduli are 2 nm independent real GEMMs;
//   - residues are held centred (|r| <= 256, exact in BF16); a chunk of KC = 256 terms
//     sums to less than 2^24, so the FP32 accumulators hold exact integers whatever the
//     signs; each chunk is reduced modulo p while the next one runs;
//   - T / P (P the product of the moduli) is the fractional part of sum_p s_p w_p with
//     s_p = u + v or u - v and w_p a 96-bit constant, so the reconstruction is a sum of
//     small times wide integers that wraps by itself, one 64 x 64 product by P and one
//     rounding. Error of a result before that rounding: 2^-bits max|A row| max|B column|
//     per term (of the scaled operands), from the rounding of the operands alone.
//
// Why: the FP64 units of this part do two FMAs per SM and cycle (1.0 TF/s measured for
// the DMMA kernel, zgemm_f64.cu); 28 BF16 products at the tensor cores' rate are some 40
// times faster. Rows that hold an infinity or NaN, and results outside the normal FP64 range,
// are multiplied entry by entry in FP64 by the reconstruction kernel.
#include "rns.cuh"
#include "launch.cuh"
#include "mpo_stage.cuh"
#include <cooperative_groups.h>
#include <cuda.h>
#include <algorithm>
#include <climits>
#include <cmath>
#include <mutex>

namespace cg = cooperative_groups;

namespace ptn {

void note_launches(int n);

namespace {

typedef __nv_bfloat16 bf16;
typedef unsigned long long u64;
typedef unsigned __int128 u128;

// ------------------------------------------------------------------ constants
constexpr int NMOD = RNS_FP64;
constexpr int MOD[NMOD] = {509, 505, 493, 481, 461, 457, 449, 433, 421, 409, 401, 397, 389, 373};
constexpr int PIECES = 5, PBITS = 11;     // |T| < 2^55 in five 11-bit pieces
constexpr int MAX_BITS = 54;
constexpr int KC = 256;                   // terms per exact FP32 sum: 256 * 255^2 < 2^24
static_assert((long)KC * 255 * 255 < (1L << 24), "chunk sums are exact in FP32");

constexpr int mod_pos(long a, int p) { return (int)(((a % p) + p) % p); }
constexpr int mod_centred(long a, int p) {
  const int r = mod_pos(a, p);
  return r > p / 2 ? r - p : r;
}
constexpr int mod_inv(long a, int p) {
  for (int x = 1; x < p; ++x)
    if (mod_pos(a, p) * (long)x % p == 1) return x;
  return 0;
}
constexpr int sqrt_minus_one(int p) {
  for (long x = 1; x < p; ++x)
    if (x * x % p == p - 1) return (int)x;
  return 0;
}

template <int NM>
struct RnsConst {
  float p[NM], inv[NM];
  float cx[NM][PIECES], cy[NM][PIECES];   // 2^(11 i) and j 2^(11 i) modulo p, centred
  unsigned wx[NM][3], wy[NM][3];          // 2^96 w_p of the real / imaginary part, low first
  u64 off_x_hi, off_y_hi;                 // 512 sum_p w_p modulo 1 (64 + 32 bits)
  unsigned off_x_lo, off_y_lo;
  u64 pm;                                 // P, top 64 bits
  int pe;                                 // floor(log2 P)
};

template <int NM>
constexpr RnsConst<NM> make_const() {
  RnsConst<NM> c{};
  u128 P = 1;
  for (int i = 0; i < NM; ++i) P *= (u128)MOD[i];
  u128 ox = 0, oy = 0;
  for (int i = 0; i < NM; ++i) {
    const int p = MOD[i];
    const int j = sqrt_minus_one(p);
    c.p[i] = (float)p;
    c.inv[i] = 1.0f / (float)p;
    long pw = 1;
    for (int q = 0; q < PIECES; ++q) {
      c.cx[i][q] = (float)mod_centred(pw, p);
      c.cy[i][q] = (float)mod_centred(pw * j, p);
      pw = (pw << PBITS) % p;
    }
    const int m = mod_inv((long)((P / (u128)p) % (u128)p), p);   // (P / p)^-1 modulo p
    const long ax = (long)m * mod_inv(2, p) % p, ay = (long)m * mod_inv(2L * j, p) % p;
    const u128 w0 = ((u128)ax << 96) / (u128)p, w1 = ((u128)ay << 96) / (u128)p;
    for (int q = 0; q < 3; ++q) {
      c.wx[i][q] = (unsigned)(w0 >> (32 * q));
      c.wy[i][q] = (unsigned)(w1 >> (32 * q));
    }
    ox += 512 * w0;
    oy += 512 * w1;
  }
  c.off_x_lo = (unsigned)ox;
  c.off_x_hi = (u64)(ox >> 32);
  c.off_y_lo = (unsigned)oy;
  c.off_y_hi = (u64)(oy >> 32);
  int e = 0;
  while ((P >> (e + 1)) != 0) ++e;
  c.pe = e;
  c.pm = (u64)(e >= 63 ? P >> (e - 63) : P << (63 - e));
  return c;
}

constexpr bool moduli_ok() {
  for (int i = 0; i < NMOD; ++i) {
    if (sqrt_minus_one(MOD[i]) == 0 || MOD[i] % 2 == 0) return false;
    for (int k = 0; k < i; ++k) {
      int a = MOD[i], b = MOD[k];
      while (b != 0) {
        const int t = a % b;
        a = b;
        b = t;
      }
      if (a != 1) return false;
    }
  }
  return true;
}
static_assert(moduli_ok(), "moduli: odd, pairwise coprime, -1 a square");

// p and 1 / p by run-time index (the GEMM's epilogue); the other kernels unroll over the
// moduli and take every constant as an immediate operand
struct ModTable {
  float p[NMOD], inv[NMOD];
};
constexpr ModTable make_table() {
  ModTable t{};
  for (int i = 0; i < NMOD; ++i) {
    t.p[i] = (float)MOD[i];
    t.inv[i] = 1.0f / (float)MOD[i];
  }
  return t;
}
__constant__ ModTable c_mod = make_table();

constexpr float MAGIC = 12582912.0f;   // 1.5 2^23: adding it rounds to an integer

// two FP32 operations in one instruction
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(reinterpret_cast<u64&>(d))
      : "l"(reinterpret_cast<u64&>(a)), "l"(reinterpret_cast<u64&>(b)), "l"(reinterpret_cast<u64&>(c)));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("add.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<u64&>(d))
      : "l"(reinterpret_cast<u64&>(a)), "l"(reinterpret_cast<u64&>(b)));
  return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 d;
  asm("mul.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<u64&>(d))
      : "l"(reinterpret_cast<u64&>(a)), "l"(reinterpret_cast<u64&>(b)));
  return d;
}
__device__ __forceinline__ float2 both(float x) { return make_float2(x, x); }

// v modulo p, centred, for two integers |v| <= 2^24 (off centre by one at most)
__device__ __forceinline__ float2 reduce_mod2(float2 v, float p, float inv) {
  const float2 q = add2(fma2(v, both(inv), both(MAGIC)), both(-MAGIC));
  return fma2(q, both(-p), v);
}

__device__ __forceinline__ int biased_exp(double x) {
  return (int)((__double_as_longlong(x) >> 52) & 0x7FF);
}

// ------------------------------------------------------------------ exponents
// A component x != 0 has the exponent e with 2^(e - 1023) <= |x| < 2^(e - 1022), subnormal
// ones below 1. Rows keep the largest e + s of their entries, s the scaling of the term, plus
// EXP_BASE: positive, so that 0 can mean a row without entries.
constexpr int EXP_BASE = 1 << 13;
constexpr int EXP_SPECIAL = 1 << 20;   // the row holds an infinity or NaN: products in FP64
constexpr int EXP_NONE = -(1 << 20);   // no entry
constexpr int TERM_DROP = -(1 << 16);  // scaling of a term that meets zeros alone

__device__ __forceinline__ int entry_exp(double2 z) {
  const int E = max(biased_exp(z.x), biased_exp(z.y));
  const u64 x = (u64)__double_as_longlong(z.x), y = (u64)__double_as_longlong(z.y);
  const u64 m = (x | y) & ((1ULL << 52) - 1);   // its top bit is that of the larger component
  const int sub = m != 0 ? 12 - __clzll((long long)m) : EXP_NONE;
  return E != 0 ? E : sub;
}

// an entry's part of its row's exponent
__device__ __forceinline__ int row_exp(double2 z, int s) {
  const int e = entry_exp(z);
  return e == 2047 ? EXP_SPECIAL : max(e + s + EXP_BASE, 0);
}

// Largest finite exponent of every term of an operand (EXP_NONE: zeros); terms k = (o, i), i <
// in, in > 1: f[o], the largest of its terms, and be[k] relative to it. A view whose rows are
// next to each other: `wpt` warps take a term, or a CTA the terms of an o; otherwise (in = 1) a
// CTA takes TERM_COLS terms (64 bytes of a row). Several operands in one launch.
// Bound: memory (the operands read once), latency where they are small.
constexpr int TERM_COLS = 4;
struct TermJob {
  RnsView v;
  int rows, kc, in;
  int *be, *f;
  int wpt, ctas;
};

struct TermJobs {
  TermJob j[RNS_TERM_JOBS];
};

__global__ void __launch_bounds__(256) k_term_exp(const TermJobs jobs, const int* skip) {
  grid_wait();
  if (skip != nullptr && *skip != 0) return;
  __shared__ int s_max[8][TERM_COLS];
  int b = blockIdx.x;
  TermJob j = jobs.j[0];
#pragma unroll
  for (int i = 1; i < RNS_TERM_JOBS; ++i)
    if (b >= j.ctas) {
      b -= j.ctas;
      j = jobs.j[i];
    }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int m = EXP_NONE;
  // entries first, first + step, ... < rows, `stride` apart: eight loads in flight
  auto take = [&](const double2* src, long stride, int first, int step) {
    for (int r = first; r < j.rows; r += 8 * step) {
      double2 z[8];
#pragma unroll
      for (int q = 0; q < 8; ++q)
        z[q] = r + q * step < j.rows ? src[(r + q * step) * stride] : make_double2(0.0, 0.0);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const bool fx = biased_exp(z[q].x) != 2047, fy = biased_exp(z[q].y) != 2047;
        m = max(m, entry_exp(make_double2(fx ? z[q].x : 0.0, fy ? z[q].y : 0.0)));
      }
    }
  };
  if (j.in > 1) {
    __shared__ int s_be[RNS_INNER_MAX];
    for (int i = warp; i < j.in; i += 8) {
      const double2* src = j.v.src + ((long)b * j.in + i) * j.v.sk;
      m = EXP_NONE;
      take(src, 1, lane, 32);
      m = __reduce_max_sync(0xffffffffu, m);
      if (lane == 0) s_be[i] = m;
    }
    __syncthreads();
    if (warp == 0) {
      m = EXP_NONE;
      for (int i = lane; i < j.in; i += 32) m = max(m, s_be[i]);
      m = __reduce_max_sync(0xffffffffu, m);
      if (lane == 0) j.f[b] = m;
      for (int i = lane; i < j.in; i += 32)
        j.be[b * j.in + i] = s_be[i] != EXP_NONE ? s_be[i] - m : EXP_NONE;
    }
  } else if (j.wpt > 0) {
    const int k = b * (8 / j.wpt) + warp / j.wpt;
    if (k < j.kc) {
      const double2* src = j.v.src + (long)k * j.v.sk;
      take(src, 1, (warp % j.wpt) * 32 + lane, 32 * j.wpt);
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if (lane == 0) s_max[warp][0] = m;
    __syncthreads();
    if (lane == 0 && warp % j.wpt == 0 && k < j.kc) {
      for (int w = 1; w < j.wpt; ++w) m = max(m, s_max[warp + w][0]);
      j.be[k] = m;
    }
  } else {
    const int k = b * TERM_COLS + (lane & (TERM_COLS - 1));
    if (k < j.kc)
      take(j.v.src + (long)k * j.v.sk, j.v.sr, warp * (32 / TERM_COLS) + lane / TERM_COLS,
           256 / TERM_COLS);
#pragma unroll
    for (int o = TERM_COLS; o < 32; o *= 2) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane < TERM_COLS) s_max[warp][lane] = m;
    __syncthreads();
    if (warp == 0 && lane < TERM_COLS && k < j.kc) {
      for (int w = 1; w < 8; ++w) m = max(m, s_max[w][lane]);
      j.be[k] = m;
    }
  }
}

// What a conversion does to the terms of its operand: nothing (t null), forms the scaling t
// and applies its inverse (`source`), or applies t (the other operand).
struct TermScale {
  const int *be, *f, *o;
  int* t;
  int in, odiv, omod;
  bool source;
};

// Powers of two that the terms [k0, k0 + kn) of the operand take, to sh (shared memory, behind a
// barrier of the caller's); the `writer` CTA of these terms leaves t for the other operand.
//   The other operand's sizes o known: largest entries a_k (other) and b_k (source) meet in a
// product of 2^S at most, S = max (a_k + b_k); the rows lose the bits by which max a + max b
// exceeds S. Every t with b_k - H <= t_k <= G - a_k, G + H = S, loses none: the one nearest to 0, so
// that operands which do not grow against each other stay as they are.
//   Not known: t from the source alone, whole pairs of bits below its largest terms.
template <int NT>
__device__ __forceinline__ void term_shifts(const TermScale& ts, int K, int k0, int kn, int* sh,
                                            bool writer) {
  if (!ts.source) {
    for (int k = threadIdx.x; k < kn; k += NT) sh[k] = ts.t[k0 + k];
    return;
  }
  constexpr int NW = NT / 32;
  __shared__ int s_top[3][NW], s_g[RNS_INNER_MAX];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (ts.o != nullptr) {
    auto other = [&](int k) { return ts.o[(k / ts.odiv) % ts.omod]; };
    int a = EXP_NONE, b = EXP_NONE, both = 2 * EXP_NONE;
    for (int k = threadIdx.x; k < K; k += NT) {
      const int ok = other(k), bk = ts.be[k];
      a = max(a, ok);
      b = max(b, bk);
      both = max(both, ok + bk);
    }
    a = __reduce_max_sync(0xffffffffu, a);
    b = __reduce_max_sync(0xffffffffu, b);
    both = __reduce_max_sync(0xffffffffu, both);
    if (lane == 0) {
      s_top[0][warp] = a;
      s_top[1][warp] = b;
      s_top[2][warp] = both;
    }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      a = max(a, s_top[0][w]);
      b = max(b, s_top[1][w]);
      both = max(both, s_top[2][w]);
    }
    const int loss = both > EXP_NONE / 2 ? a + b - both : 0;   // no common term: nothing to lose
    const int ga = a - loss / 2, hb = b - (loss - loss / 2);   // G, H
    for (int q = threadIdx.x; q < kn; q += NT) {
      const int k = k0 + q, ok = other(k), bk = ts.be[k];
      const int t = loss < 2 ? 0 : max(bk - hb, min(ga - ok, 0));
      sh[q] = ok == EXP_NONE ? TERM_DROP : -t;
      if (writer) ts.t[k] = bk == EXP_NONE ? TERM_DROP : t;
    }
    return;
  }
  const int no = K / ts.in;
  const int* f = ts.in > 1 ? ts.f : ts.be;
  auto in_pairs = [](int below) { return below & ~1; };
  int top = EXP_NONE;
  for (int o = threadIdx.x; o < no; o += NT) top = max(top, f[o]);
  top = __reduce_max_sync(0xffffffffu, top);
  if (lane == 0) s_top[0][warp] = top;
  if (ts.in > 1)
    for (int i = warp; i < ts.in; i += NW) {
      int g = EXP_NONE;
      for (int o = lane; o < no; o += 32) g = max(g, ts.be[o * ts.in + i]);
      g = __reduce_max_sync(0xffffffffu, g);
      if (lane == 0) s_g[i] = g;
    }
  __syncthreads();
#pragma unroll
  for (int w = 0; w < NW; ++w) top = max(top, s_top[0][w]);
  for (int q = threadIdx.x; q < kn; q += NT) {
    const int k = k0 + q, o = k / ts.in;
    const int t = ts.be[k] == EXP_NONE ? TERM_DROP
                  : -in_pairs(top - f[o]) - (ts.in > 1 ? in_pairs(-s_g[k - o * ts.in]) : 0);
    sh[q] = -t;
    if (writer) ts.t[k] = t;
  }
}

// pieces of T = round(x 2^(bits - e)), |x| < 2^e, e = E - 1022, as signed floats (0 where x is
// too small for one bit)
__device__ __forceinline__ void pieces_of(double x, int E, int bits, float (&f)[PIECES]) {
  const long long b = __double_as_longlong(x);
  const int Ex = (int)((b >> 52) & 0x7FF);
  u64 T = 0;
  const u64 frac = (u64)b & ((1ULL << 52) - 1);
  const u64 mant = Ex != 0 ? frac | (1ULL << 52) : frac;
  const int rs = E - max(Ex, 1) + 53 - bits;
  if (rs > 0) T = rs < 55 ? (mant + (1ULL << (rs - 1))) >> rs : 0;
  else if (mant != 0) T = mant << (-rs);
  const unsigned sign = (unsigned)((u64)b >> 32) & 0x80000000u;
#pragma unroll
  for (int i = 0; i < PIECES; ++i) {
    const unsigned q = (unsigned)(T >> (PBITS * i)) & ((1u << PBITS) - 1u);
    const float g = __uint_as_float(q | 0x4B000000u) - 8388608.0f;
    f[i] = __uint_as_float(__float_as_uint(g) ^ sign);
  }
}

// Residues of two neighbouring terms in all planes: x and y as five pieces times small
// constants, two reductions, the two terms side by side in packed FP32 operations (17 per
// modulus instead of 36: H_eff at bond 512, mixed, 360 -> 340 us with the GEMM's epilogue in
// the same form).
template <int NM>
__device__ __forceinline__ void convert_pair(const double2 (&z)[2], const int (&E)[2], int bits,
                                             bf16* __restrict__ row, long plane) {
  constexpr RnsConst<NM> c = make_const<NM>();
  float px[2][PIECES], py[2][PIECES];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    pieces_of(z[q].x, E[q], bits, px[q]);
    pieces_of(z[q].y, E[q], bits, py[q]);
  }
  float2 x[PIECES], y[PIECES];
#pragma unroll
  for (int t = 0; t < PIECES; ++t) {
    x[t] = make_float2(px[0][t], px[1][t]);
    y[t] = make_float2(py[0][t], py[1][t]);
  }
#pragma unroll
  for (int i = 0; i < NM; ++i) {
    float2 sx = x[0], sy = mul2(y[0], both(c.cy[i][0]));
#pragma unroll
    for (int t = 1; t < PIECES; ++t) {
      sx = fma2(x[t], both(c.cx[i][t]), sx);
      sy = fma2(y[t], both(c.cy[i][t]), sy);
    }
    const float2 u = reduce_mod2(add2(sx, sy), c.p[i], c.inv[i]);
    const float2 w = reduce_mod2(fma2(sy, both(-1.0f), sx), c.p[i], c.inv[i]);
    *reinterpret_cast<__nv_bfloat162*>(row + (2L * i) * plane) = __floats2bfloat162_rn(u.x, u.y);
    *reinterpret_cast<__nv_bfloat162*>(row + (2L * i + 1) * plane) =
        __floats2bfloat162_rn(w.x, w.y);
  }
}

// one entry to shared memory, asynchronously; zero (and no read) where `on` is false
__device__ __forceinline__ void load_async(double2* dst, const double2* src, bool on) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(
                   static_cast<unsigned>(__cvta_generic_to_shared(dst))),
               "l"(src), "r"(on ? 16 : 0)
               : "memory");
}

// Residue planes of a view with any strides: a CTA takes 8 rows (128 contiguous bytes per
// term of a transposed view) and part of the terms into shared memory; the CTAs of a
// cluster share the rows' terms and exchange the row maxima, so the view is read once and
// nothing is zeroed before. `have_exp`: the exponents are in e (no exchange). Bound: the
// FP32 pipe, then the writes (4 nm bytes per entry). A lane holds two neighbouring terms,
// so a warp (one row) writes 128 contiguous bytes per plane.
// Measured, 1280 x 250: 23.5 us in three launches (memset, maximum, conversion) -> 12.0.
constexpr int CR = 8;              // rows of a CTA
constexpr int CK_MAX = 1024;       // most terms of a CTA (128 KB)

template <int NM>
__global__ void __launch_bounds__(256) k_convert(const RnsView v, int R, int K, int chunk,
                                                 int* __restrict__ e, int have_exp, int bits,
                                                 bf16* __restrict__ dst, long Kp, long plane,
                                                 int* __restrict__ clear, int nclear,
                                                 const TermScale ts, const int* skip) {
  grid_wait();
  if (skip != nullptr && *skip != 0) return;   // uniform over the launch
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* tile = reinterpret_cast<double2*>(smem_raw);   // [CR][chunk + 1]
  int* shift = reinterpret_cast<int*>(tile + CR * (chunk + 1));   // of the terms
  __shared__ int s_max[CR];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool scaled = NM == RNS_FP64 && ts.t != nullptr;
  const int r0 = blockIdx.x * CR, k0 = blockIdx.y * chunk, ld = chunk + 1;
  const int kn = min(chunk, K - k0);           // terms of this CTA (the last may have fewer)
  for (int i = (blockIdx.y * gridDim.x + blockIdx.x) * 256 + tid; i < nclear;
       i += gridDim.x * gridDim.y * 256)
    clear[i] = 0;
  if (tid < CR) s_max[tid] = 0;
  if (v.sk == 1) {
    const int r = r0 + warp;
    for (int k = lane; k < chunk; k += 32)
      load_async(&tile[warp * ld + k], v.src + (long)r * v.sr + k0 + k, r < R && k < kn);
  } else {
    const int rr = tid & 7, r = r0 + rr;
    for (int k = tid >> 3; k < chunk; k += 32)
      load_async(&tile[rr * ld + k], v.src + (long)r * v.sr + (long)(k0 + k) * v.sk, r < R && k < kn);
  }
  if (scaled) term_shifts<256>(ts, K, k0, kn, shift, blockIdx.x == 0);   // meanwhile
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  const double2* row = tile + warp * ld;
  const int r = r0 + warp;
  int E;
  if (have_exp) {
    E = r < R ? e[r] : 0;
  } else {
    E = 0;
    for (int k = lane; k < kn; k += 32) E = max(E, row_exp(row[k], scaled ? shift[k] : 0));
    E = __reduce_max_sync(0xffffffffu, E);
    if (gridDim.y > 1) {
      cg::cluster_group cluster = cg::this_cluster();
      if (lane == 0) s_max[warp] = E;
      cluster.sync();
      E = lane < (int)gridDim.y ? *cluster.map_shared_rank(&s_max[warp], lane) : 0;
      E = __reduce_max_sync(0xffffffffu, E);
      cluster.sync();   // no CTA leaves while its maxima are read
    }
    if (lane == 0 && blockIdx.y == 0 && r < R) e[r] = E;
  }
  if (r >= R) return;
  const bool live = E != 0 && E != EXP_SPECIAL;
  const int kend = (int)min((long)chunk, Kp - k0);
  for (int k = 2 * lane; k < kend; k += 64) {
    double2 z[2];
    int ez[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      z[q] = live ? row[k + q] : make_double2(0.0, 0.0);
      if (v.conj) z[q].y = -z[q].y;
      ez[q] = E - EXP_BASE - (scaled && k + q < kn ? shift[k + q] : 0);
    }
    convert_pair<NM>(z, ez, bits, dst + (long)r * Kp + k0 + k, plane);
  }
}

// The exponents alone, for rows too long for a cluster (e zeroed before). Rows of the mixed
// form alone are that long: no scaling of the terms.
__global__ void __launch_bounds__(256) k_row_exp(const RnsView v, int R, int K, int* __restrict__ e,
                                                 const int* skip) {
  if (skip != nullptr && *skip != 0) return;
  __shared__ int s_max[32];
  const int rr = v.sk == 1 ? (int)threadIdx.x >> 5 : (int)threadIdx.x & 7;
  const int kk = v.sk == 1 ? (int)threadIdx.x & 31 : (int)threadIdx.x >> 3;
  if (threadIdx.x < CR) s_max[threadIdx.x] = 0;
  __syncthreads();
  const int r = blockIdx.x * CR + rr;
  int m = 0;
  if (r < R)
    for (long k = blockIdx.y * (long)CK_MAX + kk; k < min((long)K, (blockIdx.y + 1) * (long)CK_MAX); k += 32) {
      const double2 z = v.src[(long)r * v.sr + k * v.sk];
      m = max(m, row_exp(z, 0));
    }
  atomicMax(&s_max[rr], m);
  __syncthreads();
  if (threadIdx.x < CR && blockIdx.x * CR + threadIdx.x < R && s_max[threadIdx.x] > 0)
    atomicMax(&e[blockIdx.x * CR + threadIdx.x], s_max[threadIdx.x]);
}

// Views with contiguous rows of at most ROW_MAX terms: one warp finds the exponent of its
// row and converts it (the second read hits L1 / L2). Also zeroes clear[0 .. nclear) for a
// later kernel of the stream.
constexpr int ROW_MAX = 512;

template <int NM>
__global__ void __launch_bounds__(128) k_convert_rows(const RnsView v, int R, int K,
                                                      int* __restrict__ e, int bits,
                                                      bf16* __restrict__ dst, long Kp, long plane,
                                                      int* __restrict__ clear, int nclear,
                                                      const TermScale ts, const int* skip) {
  grid_wait();
  if (skip != nullptr && *skip != 0) return;
  __shared__ int shift[NM == RNS_FP64 ? ROW_MAX : 1];
  const bool scaled = NM == RNS_FP64 && ts.t != nullptr;
  if (scaled) {
    term_shifts<128>(ts, K, 0, K, shift, blockIdx.x == 0);
    __syncthreads();
  }
  for (int i = blockIdx.x * 128 + threadIdx.x; i < nclear; i += gridDim.x * 128) clear[i] = 0;
  const int lane = threadIdx.x & 31;
  const int r = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (r >= R) return;
  const double2* src = v.src + (long)r * v.sr;
  int E = 0;
  for (int k0 = lane; k0 < K; k0 += 128) {   // four loads in flight
    double2 z[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) z[q] = k0 + 32 * q < K ? src[k0 + 32 * q] : make_double2(0.0, 0.0);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      E = max(E, row_exp(z[q], scaled && k0 + 32 * q < K ? shift[k0 + 32 * q] : 0));
  }
  E = __reduce_max_sync(0xffffffffu, E);
  if (lane == 0) e[r] = E;
  const bool live = E != 0 && E != EXP_SPECIAL;
  for (int k = 2 * lane; k < Kp; k += 64) {
    double2 z[2];
    int ez[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      z[q] = (live && k + q < K) ? src[k + q] : make_double2(0.0, 0.0);
      if (v.conj) z[q].y = -z[q].y;
      ez[q] = E - EXP_BASE - (scaled && k + q < K ? shift[k + q] : 0);
    }
    convert_pair<NM>(z, ez, bits, dst + (long)r * Kp + k, plane);
  }
}

// ------------------------------------------------------------------ GEMM
constexpr int BM = 128, BK = 64;
constexpr int A_STAGE = BM * BK * 2;
constexpr int EPI_WARPS = 8;
constexpr int THREADS = 64 + 32 * EPI_WARPS;
constexpr long WAIT_LIMIT = 1L << 22;
constexpr int KB_CHUNK = KC / BK;

template <int BN>
struct Tile {
  static constexpr int B_STAGE = BN * BK * 2;
  static constexpr int STAGE = A_STAGE + B_STAGE;
  static constexpr int STAGES = BN == 256 ? 4 : 6;
  static constexpr int SMEM = STAGES * STAGE + 1024 + 256;
  static constexpr int TMEM = 2 * BN;       // two accumulators (a power of two)
  static constexpr int COLS = BN / 2;       // columns per epilogue warp
  // kind::f16 instruction descriptor: FP32 accumulate (bit 4), A and B BF16 (bits 7, 10),
  // both K-major, N >> 3 at bit 17, M >> 4 at bit 24
  static constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) |
                                    ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
  static_assert(SMEM <= 227 * 1024, "shared memory per CTA");
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(u64* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(u64* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(u64* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// bounded wait on the phase with parity `parity` that also gives up once another role
// raised the CTA's abort flag (null: none); false on expiry
__device__ __forceinline__ bool mbar_wait(u64* bar, uint32_t parity, const int* abort_flag) {
  const uint32_t a = smem_u32(bar);
  for (long it = 0; it < WAIT_LIMIT; ++it) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
    if (abort_flag != nullptr && *(volatile const int*)abort_flag) return false;
  }
  return false;
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* tm, int x, int y, int z,
                                            u64* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}

// shared-memory matrix descriptor: K-major, 128-byte swizzle (layout type 2), 8-row
// groups 1024 B apart
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr) {
  uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

__device__ __forceinline__ void umma(uint32_t tmem, uint64_t ad, uint64_t bd, uint32_t idesc,
                                     uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
      "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
      : "memory");
}

__device__ __forceinline__ void umma_commit(u64* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}

// 32 lanes x 16 columns of tensor memory
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15},"
      " [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}

__device__ __forceinline__ void tmem_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// keeps every use of v after the preceding tcgen05.wait::ld
template <int N>
__device__ __forceinline__ void after_wait(uint32_t (&v)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) asm volatile("" : "+r"(v[i]));
}

struct GemmP {
  int M, N;
  int nkb;                   // K blocks of BK
  int gx, gy, units;         // N tiles, M tiles, tiles over all planes
  unsigned short* res;       // residues + 256: [plane][M][ldr]
  long ldr, rplane;
  int* err;
  const int* skip;
};

// All 2 nm real GEMMs in one launch. A persistent CTA walks the tiles u = blockIdx.x,
// + gridDim.x, ... (N tile fastest, then M tile, then plane). Warp 0 lane 0 issues TMA
// (a ring of STAGES K blocks), warp 1 lane 0 tcgen05.mma; a chunk of KC terms fills one of
// two accumulators in tensor memory while warps 2..9 (warp w: lanes 32 (w % 4).., half of
// the columns) read the other one, reduce it modulo p and add it up in registers, so the
// drain of a chunk hides behind the next chunk's MMAs, across tiles too. Every wait is
// bounded: on expiry an error code is set, the copies in flight land and TMEM is freed; the
// reconstruction gives NaN while the code stands (ptn_device_error).
template <int BN>
__global__ void __launch_bounds__(THREADS, 1)
    k_rns_gemm(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
               const GemmP g) {
  grid_wait();
  if (g.skip != nullptr && *g.skip != 0) return;   // uniform: before any barrier or allocation
  typedef Tile<BN> T;
  extern __shared__ uint8_t smem_raw8[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw8) + 1023) &
                                             ~uintptr_t(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + T::STAGES * A_STAGE;
  u64* full = reinterpret_cast<u64*>(smem + T::STAGES * T::STAGE);
  u64* empty = full + T::STAGES;
  u64* tfull = empty + T::STAGES;    // [2] a chunk's accumulator is complete
  u64* tempty = tfull + 2;           // [2] the epilogue has read it
  uint32_t* tslot = reinterpret_cast<uint32_t*>(tempty + 2);
  int* abort_flag = reinterpret_cast<int*>(tslot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nch = (g.nkb + KB_CHUNK - 1) / KB_CHUNK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < T::STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tfull[b], 1);
      mbar_init(&tempty[b], EPI_WARPS);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tslot)),
                 "r"(T::TMEM)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tslot;

  if (warp == 0 && lane == 0) {
    // ---------------- TMA producer
    int i = 0;
    bool ok = true;
    for (int u = blockIdx.x; u < g.units && ok; u += gridDim.x) {
      const int n0 = (u % g.gx) * BN, m0 = ((u / g.gx) % g.gy) * BM, pl = u / (g.gx * g.gy);
      for (int kb = 0; kb < g.nkb; ++kb, ++i) {
        const int s = i % T::STAGES;
        if (i >= T::STAGES && !mbar_wait(&empty[s], ((uint32_t)(i / T::STAGES) & 1u) ^ 1u, abort_flag)) {
          ok = false;
          break;
        }
        mbar_expect_tx(&full[s], T::STAGE);
        tma_load_3d(sA + s * A_STAGE, &tmA, kb * BK, m0, pl, &full[s]);
        tma_load_3d(sB + s * T::B_STAGE, &tmB, kb * BK, n0, pl, &full[s]);
      }
    }
    if (!ok) {
      atomicExch(g.err, 1);
      *(volatile int*)abort_flag = 1;
      // let the copies still in flight land before the CTA retires (bounded)
      for (int q = max(0, i - T::STAGES); q < i; ++q)
        mbar_wait(&full[q % T::STAGES], (uint32_t)(q / T::STAGES) & 1u, nullptr);
    }
  } else if (warp == 1 && lane == 0) {
    // ---------------- MMA issuer
    int i = 0, ch = 0;
    bool ok = true;
    for (int u = blockIdx.x; u < g.units && ok; u += gridDim.x) {
      for (int kb = 0; kb < g.nkb; ++kb, ++i) {
        const int kin = kb % KB_CHUNK;
        const int b = ch & 1;
        if (kin == 0 && ch >= 2) {
          if (!mbar_wait(&tempty[b], ((uint32_t)(ch >> 1) & 1u) ^ 1u, abort_flag)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
        const int s = i % T::STAGES;
        if (!mbar_wait(&full[s], (uint32_t)(i / T::STAGES) & 1u, abort_flag)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a0 = smem_u32(sA + s * A_STAGE), b0 = smem_u32(sB + s * T::B_STAGE);
#pragma unroll
        for (int k = 0; k < BK / 16; ++k)
          umma(tmem + (uint32_t)(b * BN), sdesc(a0 + k * 32), sdesc(b0 + k * 32), T::IDESC,
               (kin == 0 && k == 0) ? 0u : 1u);
        umma_commit(&empty[s]);
        if (kin == KB_CHUNK - 1 || kb == g.nkb - 1) {
          umma_commit(&tfull[b]);
          ++ch;
        }
      }
    }
    if (!ok) {
      atomicExch(g.err, 2);
      *(volatile int*)abort_flag = 1;
    }
    // every MMA issued is complete before the CTA may free its tensor memory: the last
    // stage commits are waited for here (bounded)
    for (int q = max(0, i - T::STAGES); q < i; ++q)
      mbar_wait(&empty[q % T::STAGES], (uint32_t)(q / T::STAGES) & 1u, nullptr);
  } else if (warp >= 2) {
    // ---------------- epilogue
    const int quad = warp & 3, half = (warp - 2) >> 2;
    const uint32_t tl = tmem + ((uint32_t)(32 * quad) << 16) + (uint32_t)(half * T::COLS);
    int ch = 0;
    bool ok = true;
    for (int u = blockIdx.x; u < g.units && ok; u += gridDim.x) {
      const int n0 = (u % g.gx) * BN + half * T::COLS, pl = u / (g.gx * g.gy);
      const int row = ((u / g.gx) % g.gy) * BM + 32 * quad + lane;
      const float p = c_mod.p[pl >> 1], inv = c_mod.inv[pl >> 1];
      float2 acc[T::COLS / 2];
      for (int c = 0; c < nch; ++c, ++ch) {
        const int b = ch & 1;
        if (!mbar_wait(&tfull[b], (uint32_t)(ch >> 1) & 1u, abort_flag)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int c0 = 0; c0 < T::COLS; c0 += 16) {
          uint32_t v[16];
          __syncwarp();
          tmem_ld16(tl + (uint32_t)(b * BN + c0), v);
          tmem_wait_ld();
          after_wait(v);
          if (c0 + 16 == T::COLS) {
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&tempty[b]);
          }
#pragma unroll
          for (int j = 0; j < 16; j += 2) {
            const float2 r = reduce_mod2(
                make_float2(__uint_as_float(v[j]), __uint_as_float(v[j + 1])), p, inv);
            float2& sum = acc[(c0 + j) >> 1];
            sum = c == 0 ? r : add2(sum, r);
          }
        }
      }
      if (!ok) break;
      if (row < g.M) {
        unsigned short* dst = g.res + (long)pl * g.rplane + (long)row * g.ldr + n0;
#pragma unroll
        for (int c0 = 0; c0 < T::COLS; c0 += 8) {
          if (n0 + c0 >= g.N) break;
          unsigned q[4];
#pragma unroll
          for (int j = 0; j < 8; j += 2) {
            float2 r = acc[(c0 + j) >> 1];
            if (nch > 1) r = reduce_mod2(r, p, inv);
            // the low half of the magic sum's bits is the residue + 256
            r = add2(r, both(MAGIC + 256.0f));
            q[j >> 1] = __byte_perm(__float_as_uint(r.x), __float_as_uint(r.y), 0x5410);
          }
          *reinterpret_cast<uint4*>(dst + c0) = make_uint4(q[0], q[1], q[2], q[3]);
        }
      }
    }
    if (!ok && !*(volatile int*)abort_flag) {
      atomicExch(g.err, 3);
      *(volatile int*)abort_flag = 1;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(T::TMEM)
                 : "memory");
  }
}

// ------------------------------------------------------------------ reconstruction
// |F| P 2^sh as FP64 for the signed 96-bit fraction F = hi 2^-64 + lo 2^-96 of P; ok is
// cleared when the result leaves the normal range. Integer arithmetic: an FP64 operation
// costs this part as much as 64 integer ones.
__device__ __forceinline__ double finish(u64 hi, unsigned lo, u64 pm, int pe, int sh, bool& ok) {
  const u64 sign = hi & (1ULL << 63);
  if (sign) {
    lo = 0u - lo;
    hi = ~hi + (lo == 0u ? 1ULL : 0ULL);
  }
  if (hi == 0) {
    if (lo == 0) return 0.0;
    hi = (u64)lo << 32;
    lo = 0;
    sh -= 64;
  }
  const int lz = __clzll((long long)hi);
  u64 m = hi << lz;
  if (lz > 0) m |= ((u64)lo << 32) >> (64 - lz);
  u64 q = __umul64hi(m, pm);
  int x = pe + 1023 - lz + sh;      // biased exponent when q has its top bit set
  if (!(q >> 63)) {
    q <<= 1;
    --x;
  }
  const u64 r = (q >> 11) + ((q >> 10) & 1ULL);
  if (x < 1 || x > 2045) {
    ok = false;
    return 0.0;
  }
  return __longlong_as_double((long long)(sign | (((u64)x << 52) + (r - (1ULL << 52)))));
}

struct ReconP {
  int M, N, K;
  const unsigned short* res;
  long ldr, rplane;
  const int *ea, *eb;
  int sh0;                // -2 bits - 2 (1022 + EXP_BASE)
  RnsView va, vb;
  const int* err;         // device_error_word(): residues may be missing once it is set
  const int* skip;
};

__device__ __noinline__ double2 direct_product(const RnsView& va, const RnsView& vb, int K, int m,
                                               int n) {
  double2 s = make_double2(0.0, 0.0);
  for (int k = 0; k < K; ++k) {
    double2 a = va.src[(long)m * va.sr + (long)k * va.sk];
    double2 b = vb.src[(long)n * vb.sr + (long)k * vb.sk];
    if (va.conj) a.y = -a.y;
    if (vb.conj) b.y = -b.y;
    s = cfma(a, b, s);
  }
  return s;
}


// the 2 NM residues of elements n and n + 1 of a row, packed (low half first); second =
// false: of n alone. 32-bit loads where n is even.
template <int NM>
__device__ __forceinline__ void load_residues(const unsigned short* __restrict__ src, long rplane,
                                              bool second, unsigned (&ru)[NM], unsigned (&rv)[NM]) {
  if ((reinterpret_cast<uintptr_t>(src) & 3) == 0) {   // the leading dimension is even
#pragma unroll
    for (int i = 0; i < NM; ++i) {
      ru[i] = *reinterpret_cast<const unsigned*>(src + (2L * i) * rplane);
      rv[i] = *reinterpret_cast<const unsigned*>(src + (2L * i + 1) * rplane);
    }
  } else {
#pragma unroll
    for (int i = 0; i < NM; ++i) {
      const unsigned short* a = src + (2L * i) * rplane;
      const unsigned short* b = a + rplane;
      ru[i] = a[0] | (second ? (unsigned)a[1] << 16 : 0u);
      rv[i] = b[0] | (second ? (unsigned)b[1] << 16 : 0u);
    }
  }
}

// element (m, n) of the product from its residues (low or high half: q = 0 or 1)
template <int NM>
__device__ __forceinline__ double2 element(const ReconP& g, int m, int n, int q,
                                           const unsigned (&ru)[NM], const unsigned (&rv)[NM]) {
  constexpr RnsConst<NM> c = make_const<NM>();
  const int Ea = g.ea[m], Eb = g.eb[n];
  u64 x0 = 0, x1 = 0, y0 = 0, y1 = 0;
  unsigned x2 = 0, y2 = 0;
#pragma unroll
  for (int i = 0; i < NM; ++i) {
    const unsigned u = q ? ru[i] >> 16 : ru[i] & 0xFFFFu, v = q ? rv[i] >> 16 : rv[i] & 0xFFFFu;
    const unsigned s = u + v, d = u - v + 512u;
    x0 += (u64)s * c.wx[i][0];
    x1 += (u64)s * c.wx[i][1];
    x2 += s * c.wx[i][2];
    y0 += (u64)d * c.wy[i][0];
    y1 += (u64)d * c.wy[i][1];
    y2 += d * c.wy[i][2];
  }
  x1 += x0 >> 32;
  y1 += y0 >> 32;
  const unsigned xl = (unsigned)x0, yl = (unsigned)y0;
  u64 xh = x1 + ((u64)x2 << 32), yh = y1 + ((u64)y2 << 32);
  xh -= c.off_x_hi + (xl < c.off_x_lo ? 1ULL : 0ULL);
  yh -= c.off_y_hi + (yl < c.off_y_lo ? 1ULL : 0ULL);
  if (*g.err != 0) return make_double2(__longlong_as_double(-1LL), __longlong_as_double(-1LL));
  bool ok = Ea != EXP_SPECIAL && Eb != EXP_SPECIAL;
  double2 z = make_double2(0.0, 0.0);
  if (ok && Ea != 0 && Eb != 0) {
    const int sh = Ea + Eb + g.sh0;
    z.x = finish(xh, xl - c.off_x_lo, c.pm, c.pe, sh, ok);
    z.y = finish(yh, yl - c.off_y_lo, c.pm, c.pe, sh, ok);
  }
  if (!ok) z = direct_product(g.va, g.vb, g.K, m, n);
  return z;
}

// alpha z + beta y as the DMMA kernel forms it. Not inlined: alpha = 1, beta = 0 needs it for
// infinities and NaNs alone (0 * inf), and an FP64 operation that the compiler hoists out of
// the rare branch costs every element 64 cycles of a sub-partition.
__device__ __noinline__ double2 scale_add(double2 alpha, double2 z, double2 beta, const double2* y) {
  z = cmul(alpha, z);
  return y != nullptr ? cadd(z, cmul(beta, *y)) : z;
}

__device__ __forceinline__ bool not_finite(double2 z) {
  return biased_exp(z.x) == 2047 || biased_exp(z.y) == 2047;
}

// Bound: latency of the loads (all residues of a pair are fetched ahead: fewer in flight and
// more warps was slower), then the integer pipe (about 10 operations per residue pair).
// Measured, 1024 x 512, 11 moduli: 22 us while an alpha z was formed speculatively for every
// element -> 14.
template <int NM>
__global__ void __launch_bounds__(256) k_reconstruct(const ReconP g, double2 alpha, double2 beta,
                                                     int plain, int add,
                                                     double2* __restrict__ out, long ldc) {
  grid_wait();
  if (g.skip != nullptr && *g.skip != 0) return;
  const int np = (g.N + 1) >> 1;
  const long total = (long)g.M * np;
  for (long idx = blockIdx.x * 256L + threadIdx.x; idx < total; idx += gridDim.x * 256L) {
    const int m = (int)(idx / np), n = 2 * (int)(idx % np);
    unsigned ru[NM], rv[NM];
    load_residues<NM>(g.res + (long)m * g.ldr + n, g.rplane, n + 1 < g.N, ru, rv);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      if (n + q >= g.N) break;
      double2 z = element<NM>(g, m, n + q, q, ru, rv);
      double2* o = out + (long)m * ldc + n + q;
      if (!plain || not_finite(z)) z = scale_add(alpha, z, beta, add ? o : nullptr);
      *o = z;
    }
  }
}

// Reconstruction fused with the MPO stage (mpo_stage.cuh): the product's element
// ((x, p / pin), (p % pin, y)) is stage input (x, p, y), put together straight into the
// shared-memory rows of the stage; the stage output goes to `out` and the exponents of the
// rows it forms as the next operand to e2 (zeroed before). by_x false: rows (q % eq, y);
// true: rows (x, q / eq). t2 (or null): the scaling of that operand's terms. One CTA per (x, 128-wide y chunk), of STAGE_Y threads, or twice as
// many where the CTAs alone leave too few warps in flight for the chain of loads and wide
// integer sums. Saves writing and reading the product in FP64 and a maximum pass over the
// stage output.
template <int NM>
__global__ void __launch_bounds__(2 * STAGE_Y)
    k_reconstruct_stage(const ReconP g, const double2* __restrict__ w, long ldq, long ldp, int P,
                        int pin, int Q, int Y, double2* __restrict__ out, int* __restrict__ e2,
                        const int* __restrict__ t2, int eq, int by_x) {
  grid_wait();
  if (g.skip != nullptr && *g.skip != 0) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* sin = reinterpret_cast<double2*>(smem_raw);
  double2* sval = sin + (size_t)P * STAGE_Y;
  int* sidx = reinterpret_cast<int*>(sval + (size_t)P * Q);
  __shared__ int scount[STAGE_MAX];
  const int x = blockIdx.y, y0 = blockIdx.x * STAGE_Y, ty = threadIdx.x;
  const int na = by_x ? Q / eq : eq, nb = by_x ? eq : Q / eq;
  const bool scaled = NM == RNS_FP64 && t2 != nullptr;
  __shared__ int s_t2[STAGE_MAX];
  if (scaled && !by_x && ty < nb) s_t2[ty] = t2[(long)x * nb + ty];
  stage_load_w(w, ldq, ldp, P, Q, sval);
  const int pair = 2 * (ty & 63);
  for (int p = ty >> 6; p < P; p += blockDim.x / 64) {
    const int y = y0 + pair;
    if (y < Y) {
      const int m = x * (P / pin) + p / pin, n = (p % pin) * Y + y;
      unsigned ru[NM], rv[NM];
      load_residues<NM>(g.res + (long)m * g.ldr + n, g.rplane, y + 1 < Y, ru, rv);
      const double2 one = make_double2(1.0, 0.0);
#pragma unroll
      for (int q = 0; q < 2; ++q)
        if (y + q < Y) {
          double2 z = element<NM>(g, m, n + q, q, ru, rv);
          if (not_finite(z)) z = scale_add(one, z, one, nullptr);
          sin[p * STAGE_Y + pair + q] = z;
        }
    }
  }
  __syncthreads();
  stage_compact(P, Q, sval, sidx, scount);
  __syncthreads();
  const int yl = ty & (STAGE_Y - 1), y = y0 + yl;
  for (int a = ty / STAGE_Y; a < na; a += blockDim.x / STAGE_Y) {
    int E = 0;
    if (y < Y)
      for (int b = 0; b < nb; ++b) {
        const int q = by_x ? a * eq + b : b * eq + a;
        const double2 z = stage_row(q, P, sin + yl, sval, sidx, scount);
        out[((long)x * Q + q) * Y + y] = z;
        E = max(E, row_exp(z, !scaled ? 0 : by_x ? t2[(long)b * Y + y] : s_t2[b]));
      }
    if (by_x) {
      E = __reduce_max_sync(0xffffffffu, E);
      if ((ty & 31) == 0 && E > 0) atomicMax(&e2[x * na + a], E);
    } else if (E > 0) {
      int* dst = e2 + (long)a * Y + y;
      if (*(volatile int*)dst < E) atomicMax(dst, E);
    }
  }
}

// ------------------------------------------------------------------ tensor maps
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault,
                                         &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(f);
  });
  return fn;
}

// map over the planes [2 nm][rows][Kp] of logical extent (kc, rows, 2 nm), box (BK,
// box_rows, 1): terms beyond kc and rows beyond the last read as zero
bool make_map(CUtensorMap* out, const RnsOperand& o, int box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return false;
  cuuint64_t dims[3] = {(cuuint64_t)o.kc, (cuuint64_t)o.rows, (cuuint64_t)(2 * o.nm)};
  cuuint64_t strides[2] = {(cuuint64_t)o.Kp * 2, (cuuint64_t)o.plane() * 2};
  cuuint32_t box[3] = {(cuuint32_t)BK, (cuuint32_t)box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  return fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, o.p, dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

long residue_ld(long N) { return (N + 7) / 8 * 8; }

template <int BN>
ptn_status launch_gemm(const RnsOperand& A, const RnsOperand& B, GemmP g, cudaStream_t st) {
  CUtensorMap ma, mb;
  if (!make_map(&ma, A, BM) || !make_map(&mb, B, BN)) {
    set_error("rns_gemm: cuTensorMapEncodeTiled failed");
    return PTN_CUDA_ERROR;
  }
  static std::once_flag once;
  static cudaError_t attr = cudaSuccess;
  std::call_once(once, [] {
    attr = cudaFuncSetAttribute(k_rns_gemm<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                Tile<BN>::SMEM);
  });
  PTN_CUDA_TRY(attr);
  g.gx = (g.N + BN - 1) / BN;
  g.gy = (g.M + BM - 1) / BM;
  const long units = (long)g.gx * g.gy * 2 * A.nm;
  PTN_CHECK_ARG(units <= INT_MAX / 2, "rns_gemm: too many tiles");
  g.units = (int)units;
  const int grid = (int)std::min<long>(units, num_sms());
  PTN_CUDA_TRY(launch(k_rns_gemm<BN>, dim3(grid), dim3(THREADS), Tile<BN>::SMEM, st, ma, mb, g));
  PTN_LAUNCH_CHECK();
  return PTN_OK;
}

// cycles of a launch with N tiles of bn columns: whole turns of the SMs; per tile and 16 terms
// what the SM takes to read both operand tiles from L2 (64 bytes a cycle: 192, 128 and 96
// cycles for 256, 128 and 64 columns; the MMAs themselves take half a cycle per column),
// and a fixed cost per tile. Measured, M 2048, N 5120, K 1024: 300 us, 190 cycles per 16 terms
// of a 128 x 256 tile.
double tile_cost(int bn, long M, long N, long K, int planes) {
  const long units = ((N + bn - 1) / bn) * ((M + BM - 1) / BM) * planes;
  const long turns = (units + num_sms() - 1) / num_sms();
  const double k16 = (double)((K + 15) / 16);
  return turns * (k16 * (64.0 + bn / 2.0) + 300.0 + bn);
}

constexpr double plog2(int nm) {
  double s = 1.0;   // log2 of the product, by halving
  double l = 0.0;
  for (int i = 0; i < nm; ++i) {
    s *= MOD[i];
    while (s >= 2.0) {
      s *= 0.5;
      l += 1.0;
    }
  }
  return l;         // floor(log2 P)
}

}  // namespace

size_t rns_plane_bytes(long rows, long kc, int nm) {
  return (size_t)(2 * nm) * rows * ((kc + 7) / 8 * 8) * sizeof(bf16);
}

size_t rns_out_bytes(long M, long N, int nm) {
  return (size_t)(2 * nm) * M * residue_ld(N) * sizeof(unsigned short);
}

RnsOperand rns_operand(void* planes, void* exps, long rows, long kc, int nm) {
  RnsOperand o;
  o.p = static_cast<bf16*>(planes);
  o.e = static_cast<int*>(exps);
  o.rows = (int)rows;
  o.kc = (int)kc;
  o.nm = nm;
  o.Kp = (kc + 7) / 8 * 8;
  return o;
}

// |sum of K terms| <= K 2^(2 bits + 1) has to stay below 0.49 P; 0.49 P > 2^(floor(log2 P) - 2)
int rns_bits(long K, int nm) {
  int lk = 0;
  while ((1L << lk) < K) ++lk;
  const int room = (int)plog2(nm) - 2 - 1 - lk;
  const int bits = std::min(MAX_BITS, room / 2);
  return bits >= (nm == RNS_FP64 ? 53 : 39) ? bits : 0;
}

// The fixed cost of the path (exponents, conversions, planes, reconstruction: 16 us for a single
// GEMM) meets the DMMA kernel between 1e6 and 2e6 complex products, that of a Lanczos step
// (operands of the operator converted once) at 1e6. Measured, the GEMMs of H_eff at bond D and
// MPO bond 5 alone (first / second, DMMA -> residues):
//   D = 48: 14.2 -> 16.3, 24.9 -> 20.8 us;  56: 20.2 -> 16.6, 24.2 -> 22.6;  64: 30.1 -> 16.8,
//   28.3 -> 22.7;  128: 184 -> 26, 217 -> 27;  256: 1417 -> 58, 1456 -> 52
// whole calls: H_eff at D = 48 44.5 -> 40.5 us, 64 64.7 -> 42.5; environment steps at 48 37.3 ->
// 40.4, 56 47.5 -> 42; and a Lanczos step:
//   D = 48: 56 -> 42 us;  64: 77 -> 44;  128: 425 -> 59;  256: 2908 -> 120
bool rns_wanted(long M, long N, long K) {
  if (std::min(M, std::min(N, K)) < 32 || M > INT_MAX / 2 || N > INT_MAX / 2) return false;
  return (double)M * N * K >= 1.0e6 && rns_bits(K, RNS_FP64) != 0;
}

template <int NM>
static ptn_status launch_convert(const RnsView& v, const RnsOperand& d, bool have_exp, int bits,
                                 int* clear, int nclear, const TermScale& ts, const int* skip,
                                 cudaStream_t st) {
  static std::once_flag once;
  static cudaError_t attr = cudaSuccess;
  std::call_once(once, [] {
    attr = cudaFuncSetAttribute(k_convert<NM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                CR * (CK_MAX + 1) * (int)sizeof(double2) + CK_MAX * (int)sizeof(int));
  });
  PTN_CUDA_TRY(attr);
  // terms per CTA, multiples of 64: enough CTAs for the chip, and at most 256 terms (33 KB, six
  // CTAs per SM: an environment step at bond 1024 takes 1.84 ms with up to 1024 terms and two
  // CTAs per SM, 1.71 so), while at most 8 CTAs share a row where the maxima are exchanged
  const long groups = (d.rows + CR - 1) / CR;
  const long blocks64 = (d.kc + 63) / 64;
  long parts = std::max(std::min(2L * num_sms() / groups, blocks64), ((long)d.kc + 255) / 256);
  if (!have_exp) parts = std::min(parts, 8L);
  const long chunk = (blocks64 + parts - 1) / parts * 64;
  parts = (d.kc + chunk - 1) / chunk;
  if (chunk > CK_MAX) {   // longer than a cluster takes: the exponents in a pass of their own
    PTN_CUDA_TRY(cudaMemsetAsync(d.e, 0, (size_t)d.rows * sizeof(int), st));
    const dim3 ge((unsigned)groups, (unsigned)((d.kc + CK_MAX - 1) / CK_MAX));
    PTN_CHECK_ARG(ge.y <= 65535, "rns_convert: too many columns");
    PTN_CHECK_ARG(ts.t == nullptr, "rns_convert: rows too long for scaled terms");
    k_row_exp<<<ge, 256, 0, st>>>(v, d.rows, d.kc, d.e, skip);
    PTN_LAUNCH_CHECK();
    note_launches(1);
    return launch_convert<NM>(v, d, true, bits, clear, nclear, ts, skip, st);
  }
  PTN_CHECK_ARG(parts <= 65535, "rns_convert: too many columns");
  LaunchShape shape{dim3((unsigned)groups, (unsigned)parts), dim3(256),
                    CR * (size_t)(chunk + 1) * sizeof(double2) + chunk * sizeof(int)};
  if (!have_exp) shape.cluster = dim3(1, (unsigned)parts, 1);
  PTN_CUDA_TRY(launch_shape(k_convert<NM>, shape, st, v, d.rows, d.kc, (int)chunk, d.e,
                            have_exp ? 1 : 0, bits, d.p, d.Kp, d.plane(), clear, nclear, ts, skip));
  note_launches(1);
  return PTN_OK;
}

template <int NM>
static ptn_status convert(const RnsView& v, const RnsOperand& d, bool have_exp, int bits,
                          int* clear, int nclear, const TermScale& ts, const int* skip,
                          cudaStream_t st) {
  if (v.sk != 1 || have_exp || d.kc > ROW_MAX)
    return launch_convert<NM>(v, d, have_exp, bits, clear, nclear, ts, skip, st);
  PTN_CUDA_TRY(launch(k_convert_rows<NM>, dim3((d.rows + 3) / 4), dim3(128), 0, st, v, d.rows,
      d.kc, d.e, bits, d.p, d.Kp, d.plane(), clear, nclear, ts, skip));
  PTN_LAUNCH_CHECK();
  note_launches(1);
  return PTN_OK;
}

ptn_status rns_convert(const RnsView& v, const RnsOperand& d, bool have_exp, const int* skip,
                       cudaStream_t st, int* clear, int nclear, const RnsTerms* terms, bool source) {
  const int bits = rns_bits(d.kc, d.nm);
  PTN_CHECK_ARG(bits != 0, "rns_convert: products of %d terms are too long", d.kc);
  TermScale ts{};
  if (terms != nullptr)
    ts = TermScale{terms->be, terms->f, terms->o, terms->t, terms->in, terms->odiv, terms->omod,
                   source};
  switch (d.nm) {
    case RNS_FP64: return convert<RNS_FP64>(v, d, have_exp, bits, clear, nclear, ts, skip, st);
    case RNS_MIXED_ENV:
      return convert<RNS_MIXED_ENV>(v, d, have_exp, bits, clear, nclear, ts, skip, st);
    default: return convert<RNS_MIXED>(v, d, have_exp, bits, clear, nclear, ts, skip, st);
  }
}

ptn_status rns_term_exps(const RnsTermsOf* of, int n, const int* skip, cudaStream_t st) {
  TermJobs jobs = {};
  int ctas = 0;
  for (int i = 0; i < n; ++i) {
    TermJob& j = jobs.j[i];
    j = TermJob{of[i].v, of[i].rows, of[i].kc, of[i].in, of[i].be, of[i].f, 0, 0};
    PTN_CHECK_ARG(j.in == 1 || (j.v.sr == 1 && j.kc % j.in == 0), "rns_term_exps: bad layout");
    // warps of a term: up to four rows per lane
    j.wpt = j.v.sr != 1 ? 0 : j.rows <= 128 ? 1 : j.rows <= 256 ? 2 : j.rows <= 512 ? 4 : 8;
    const int per = j.in > 1 ? j.in : j.wpt == 0 ? TERM_COLS : 8 / j.wpt;
    j.ctas = (j.kc + per - 1) / per;
    ctas += j.ctas;
  }
  PTN_CUDA_TRY(launch(k_term_exp, dim3(ctas), dim3(256), 0, st, jobs, skip));
  note_launches(1);
  return PTN_OK;
}

// the integer products of all planes -> res, and what their reconstruction needs
static ptn_status multiply(const RnsOperand& A, const RnsView& va, const RnsOperand& B,
                           const RnsView& vb, void* res, const int* skip, cudaStream_t st,
                           ReconP* r) {
  const int M = A.rows, N = B.rows, K = A.kc;
  PTN_CHECK_ARG(M > 0 && N > 0 && K > 0 && B.kc == K && A.nm == B.nm, "rns_gemm: bad operands");
  const int bits = rns_bits(K, A.nm);
  PTN_CHECK_ARG(bits != 0, "rns_gemm: products of %d terms are too long", K);
  GemmP g;
  g.M = M;
  g.N = N;
  g.nkb = (K + BK - 1) / BK;
  g.gx = g.gy = g.units = 0;
  g.res = static_cast<unsigned short*>(res);
  g.ldr = residue_ld(N);
  g.rplane = (long)M * g.ldr;
  g.err = device_error_word();
  g.skip = skip;
  PTN_CHECK_ARG(g.err != nullptr, "rns_gemm: error flag lookup failed");
  const int planes = 2 * A.nm;
  const int prof = prof_begin(st, PROF_TC_GEMM, 8.0 * M * (double)N * K,
                              2.0 * planes * ((double)M * K + (double)N * K + (double)M * N));
  const double c64 = tile_cost(64, M, N, K, planes), c128 = tile_cost(128, M, N, K, planes),
               c256 = tile_cost(256, M, N, K, planes);
  if (c256 <= c128 && c256 <= c64) PTN_TRY(launch_gemm<256>(A, B, g, st));
  else if (c128 <= c64) PTN_TRY(launch_gemm<128>(A, B, g, st));
  else PTN_TRY(launch_gemm<64>(A, B, g, st));
  prof_end(st, prof);
  note_launches(1);
  r->M = M;
  r->N = N;
  r->K = K;
  r->res = g.res;
  r->ldr = g.ldr;
  r->rplane = g.rplane;
  r->ea = A.e;
  r->eb = B.e;
  r->sh0 = -2 * bits - 2 * (1022 + EXP_BASE);
  r->va = va;
  r->vb = vb;
  r->err = g.err;
  r->skip = skip;
  return PTN_OK;
}

ptn_status rns_gemm(const RnsOperand& A, const RnsView& va, const RnsOperand& B, const RnsView& vb,
                    double2 alpha, double2 beta, double2* out, long ldc, void* res,
                    const int* skip, cudaStream_t st) {
  ReconP r;
  PTN_TRY(multiply(A, va, B, vb, res, skip, st, &r));
  const long pairs = (long)r.M * ((r.N + 1) / 2);
  const int blocks = (int)std::min<long>((pairs + 255) / 256, 16L * num_sms());
  auto kernel = A.nm == RNS_FP64 ? k_reconstruct<RNS_FP64>
                : A.nm == RNS_MIXED_ENV ? k_reconstruct<RNS_MIXED_ENV> : k_reconstruct<RNS_MIXED>;
  const int add = beta.x != 0.0 || beta.y != 0.0;
  const int plain = !add && alpha.x == 1.0 && alpha.y == 0.0;
  PTN_CUDA_TRY(launch(kernel, dim3(blocks), dim3(256), 0, st, r, alpha, beta, plain, add, out, ldc));
  note_launches(1);
  return PTN_OK;
}

template <int NM>
static ptn_status launch_stage(const ReconP& r, const RnsStage& s, cudaStream_t st) {
  static std::once_flag once;
  static cudaError_t attr = cudaSuccess;
  std::call_once(once, [] {
    attr = cudaFuncSetAttribute(k_reconstruct_stage<NM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)stage_smem(STAGE_MAX, STAGE_MAX));
  });
  PTN_CUDA_TRY(attr);
  const dim3 grid((s.Y + STAGE_Y - 1) / STAGE_Y, s.X);
  // measured, 250 x 256: 30 -> 22 us with 256 threads (500 CTAs); 1024 x 1024 (8192 CTAs):
  // an environment step 2.09 -> 2.16 ms
  const int threads = (long)grid.x * grid.y < 16L * num_sms() ? 2 * STAGE_Y : STAGE_Y;
  PTN_CUDA_TRY(launch(k_reconstruct_stage<NM>, dim3(grid), dim3(threads), stage_smem(s.P, s.Q), st,
      r, s.w, s.ldq, s.ldp, s.P, s.pin, s.Q, s.Y, s.out, s.e2, s.t2, s.eq, s.by_x ? 1 : 0));
  PTN_LAUNCH_CHECK();
  note_launches(1);
  return PTN_OK;
}

ptn_status rns_gemm_stage(const RnsOperand& A, const RnsView& va, const RnsOperand& B,
                          const RnsView& vb, const RnsStage& s, void* res, const int* skip,
                          cudaStream_t st) {
  PTN_CHECK_ARG(s.P <= STAGE_MAX && s.Q <= STAGE_MAX, "MPO stage: chi*d must be <= 64 (got %d, %d)",
                s.P, s.Q);
  PTN_CHECK_ARG(s.X <= 65535, "MPO stage: X too large");
  ReconP r;
  PTN_TRY(multiply(A, va, B, vb, res, skip, st, &r));
  switch (A.nm) {
    case RNS_FP64: return launch_stage<RNS_FP64>(r, s, st);
    case RNS_MIXED_ENV: return launch_stage<RNS_MIXED_ENV>(r, s, st);
    default: return launch_stage<RNS_MIXED>(r, s, st);
  }
}

}  // namespace ptn
