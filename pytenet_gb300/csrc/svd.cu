// Thin singular value decomposition of a complex128 matrix: the per-block kernel of
// block_sparse_svd (pytenet/block_sparse_util.py:244-330, which calls
// numpy.linalg.svd(full_matrices=False) per quantum-number block) and so of the
// two-site splits (pytenet/bond_ops.py:41-53, pytenet/mps.py:538-568).
//
// Method: one-sided Jacobi (Hestenes) in FP64. The columns of W (A, or A^H when A
// is wide, so that W is p x r with p >= r) are orthogonalised pairwise: for a pair
// (j, k) with Gram entries a = |w_j|^2, b = |w_k|^2, c = w_j^H w_k = |c| e^{i phi},
// w_k is first turned by e^{-i phi} (which makes the pair's Gram entry real) and
// then the real Jacobi rotation with zeta = (b - a) / (2 |c|),
// t = sign(zeta) / (|zeta| + sqrt(1 + zeta^2)), cs = 1 / sqrt(1 + t^2), sn = cs t
// zeroes it: w_j <- cs w_j - sn w_k, w_k <- sn w_j + cs w_k. The same unitary column
// operations accumulate in V (r x r, starting at I). Pairs follow the round-robin
// (circle) order, r/2 disjoint pairs per round; a sweep is r - 1 rounds; sweeps repeat
// until no pair has |c| > tol sqrt(a b) (tol = p * eps), at most MAX_SWEEPS of them.
// Then s_j = |w_j|, the columns are sorted by decreasing s (ties by index, LAPACK's
// order), U = W / s, and A = U diag(s) V^H (for a wide A the roles of U and V swap).
//
// From PRE_MIN columns on, the sweeps start from the singular vectors found by the same
// iteration in FP32 (mixed-precision Jacobi: Gao, Ma and Shao 2022): V32 is made unitary in
// FP64 by a Newton-Schulz step and then improved twice for all pairs at once by GEMMs: with
// G = W^H W, W = A V, the first-order rotation V (I + X), X_ij = G_ij / (G_jj - G_ii), leaves
// the square of the off-diagonal part (pairs too close for that are left to the sweeps), and
// two more Newton-Schulz steps make it unitary. The FP64 sweeps, whose stopping rule and so
// whose accuracy stay as they are, then run only if the Gram matrix of the result shows a pair
// that the rule would rotate: none or one sweep instead of nine or ten.
// What bounds the iteration: an FP64 instruction of a warp takes 64 cycles of its
// sub-partition; the FP32 sweeps cost only their rounds' latency (sums, rotation,
// cluster barrier).
//
// Singular vectors of one singular value are unique only up to a phase (or a
// unitary mix for repeated values): they need not equal LAPACK's, while the
// singular values, the products U diag(s) V^H and every quantity built from a
// truncated split agree to rounding.
//
// One cluster of up to 16 CTAs per matrix: a round's pairs are spread over the CTAs, four
// warps to a pair; the columns stay in global memory (L2), in the FP32 sweeps in shared memory
// where they fit; a cluster barrier ends a round.
// Measured, 128 x 96: 75.6 ms (one CTA, FP64 sweeps only) -> 2.40 ms with FP32 sweeps through
// L2 (1.53 of it) -> 1.83 ms (FP32 sweeps 0.96, GEMMs 0.25, one FP64 sweep 0.57) -> 1.31 ms
// (the last check on a Gram matrix).
#include "ptn_common.cuh"
#include "fp64_seed.cuh"
#include <cooperative_groups.h>
#include <algorithm>
#include <mutex>

namespace cg = cooperative_groups;

namespace ptn {

void note_launches(int n);

namespace {

constexpr int GROUP = 128;        // threads that share a pair
constexpr int NGROUP = 4;         // groups per CTA
constexpr int ST = GROUP * NGROUP;
constexpr int MAX_SWEEPS = 60;
constexpr int PRE_SWEEPS = 15;    // at most that many FP32 sweeps
constexpr int PRE_MIN = 32;       // columns from which the FP32 sweeps pay
constexpr int NS = 5;             // Newton-Schulz steps: one, and two after each refinement
// Largest first-order rotation times the column count, by step: |X| <= X_NORM, so V is off
// unitary by X_NORM^2 at most, and every Newton-Schulz step takes an error e to 0.75 e^2
// (0.1: 1e-2 -> 8e-5 -> 4e-9; 1e-3: 1e-6 -> 8e-13 -> below rounding).
constexpr int REFINE = 2;
constexpr double X_NORM[REFINE] = {0.1, 1e-3};
constexpr int REG = 4;            // column entries a thread keeps in registers
constexpr int RANGE = 200;        // binary orders of the largest entry that need no shift: its square, and those of
                                  // columns 2^300 below it, are normal numbers

template <typename T>
struct Cplx;
template <>
struct Cplx<double> {
  typedef double2 type;
};
template <>
struct Cplx<float> {
  typedef float2 type;
};

// four values summed over the warp with seven additions: value q ends in the lanes with
// (lane & 3) == q
template <typename T>
__device__ __forceinline__ T warp_sum4(T v0, T v1, T v2, T v3) {
  const int lane = threadIdx.x & 31;
  const bool h1 = lane & 1, h2 = lane & 2;
  // lanes exchange the half they do not keep
  const T a = (h1 ? v1 : v0) + __shfl_xor_sync(0xffffffffu, h1 ? v0 : v1, 1);
  const T b = (h1 ? v3 : v2) + __shfl_xor_sync(0xffffffffu, h1 ? v2 : v3, 1);
  T c = (h2 ? b : a) + __shfl_xor_sync(0xffffffffu, h2 ? a : b, 2);
  c += __shfl_xor_sync(0xffffffffu, c, 4);
  c += __shfl_xor_sync(0xffffffffu, c, 8);
  c += __shfl_xor_sync(0xffffffffu, c, 16);
  return c;
}

// Rotation of a pair: x' = cs x - g y, y' = sn x + h y
template <typename T>
struct Rot {
  T cs, sn, gr, gi, hr, hi;
  int on;
};

__device__ __forceinline__ float fast_sqrt(float x) {
  float y;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// off: |c| / sqrt(a b) as far as FP32 tells. FP32 form, with approximate divisions and square
// roots (a few units of the last place, which V32 is off unitary by anyway).
__device__ __forceinline__ Rot<float> rotation(float aa, float bb, float cr, float ci, float tol,
                                               float& off) {
  Rot<float> R;
  R.on = 0;
  off = 0.0f;
  // columns below 1e-15 of the largest entry: beyond what FP32 resolves (and their products
  // near the end of its range)
  if (!(aa > 1e-30f && bb > 1e-30f)) return R;
  const float mx = fmaxf(fabsf(cr), fabsf(ci)), ab = fast_sqrt(aa) * fast_sqrt(bb);
  if (!(mx > 0.5f * tol * ab)) return R;
  const float im = __fdividef(1.0f, mx), ur = cr * im, ui = ci * im;
  const float u2 = ur * ur + ui * ui, ul = rsqrtf(u2);
  const float ac = mx * u2 * ul;
  off = __fdividef(ac, ab);
  R.on = ac > tol * ab;
  if (!R.on) return R;
  const float pr = ur * ul, pi = -ui * ul;
  const float z = __fdividef(bb - aa, 2.0f * ac);
  const float t = __fdividef(copysignf(1.0f, z), fabsf(z) + fast_sqrt(1.0f + z * z));
  R.cs = rsqrtf(1.0f + t * t);
  R.sn = R.cs * t;
  R.gr = R.sn * pr;
  R.gi = R.sn * pi;
  R.hr = R.cs * pr;
  R.hi = R.cs * pi;
  return R;
}

__device__ __forceinline__ int exp_of(double x) {
  return (int)((__double_as_longlong(x) >> 52) & 0x7FF) - 1023;
}

// x 2^-h as a float (0 below, infinity above its range), integer work only
__device__ __forceinline__ float scaled_float(double x, int h) {
  const long long b = __double_as_longlong(x);
  const int e = (int)((b >> 52) & 0x7FF) - h - 1023 + 127;
  const unsigned sign = (unsigned)(b >> 32) & 0x80000000u;
  if (((b >> 52) & 0x7FF) == 0 || e <= 0) return __uint_as_float(sign);
  if (e >= 255) return __uint_as_float(sign | 0x7F800000u);
  return __uint_as_float(sign | ((unsigned)e << 23) | ((unsigned)(b >> 29) & 0x7FFFFFu));
}

// FP64 throughout: columns of very different size, or near the lower end of the range. The
// Gram entries are squares already: nothing here squares them again.
__device__ __noinline__ Rot<double> rotation_fp64(double aa, double bb, double cr, double ci,
                                                  double tol, float& off) {
  Rot<double> R;
  const double ac = hypot(cr, ci), ab = sqrt(aa) * sqrt(bb);
  R.on = ac > 0.0 && ac > tol * ab;
  off = R.on ? (float)fmax(ac / ab, 1e-30) : 0.0f;
  if (!R.on) return R;
  const double pr = cr / ac, pi = -ci / ac;
  const double z = (bb - aa) / (2.0 * ac);
  const double t = copysign(1.0, z) / (fabs(z) + hypot(1.0, z));
  R.cs = 1.0 / sqrt(1.0 + t * t);
  R.sn = R.cs * t;
  R.gr = R.sn * pr;
  R.gi = R.sn * pi;
  R.hr = R.cs * pr;
  R.hi = R.cs * pi;
  return R;
}

// FP64 form, by a whole warp (all lanes get the result). The angle and the phase need only
// FP32 accuracy (an angle off by 1e-7 leaves 1e-7 of c, as good as another sweep); the
// rotation itself is unitary to FP64 accuracy: lane 0 forms cs = (1 + t^2)^-1/2, lane 1 the
// modulus of the FP32 phase, with the same instructions. FP64 divisions and square roots
// would take 64 cycles for every one of their dozens of steps.
__device__ __forceinline__ Rot<double> rotation(double aa, double bb, double cr, double ci,
                                                double tol, float& off) {
  Rot<double> R;
  const int ea = exp_of(aa), eb = exp_of(bb), h = (ea + eb) >> 1;
  R.on = 0;
  off = 0.0f;
  if (ea == 1024 || eb == 1024) return R;            // overflow, NaN: left alone
  if (ea < -960 || eb < -960) return rotation_fp64(aa, bb, cr, ci, tol, off);
  const float fr = scaled_float(cr, h), fi = scaled_float(ci, h);
  const float ab = scaled_float(aa, ea) * scaled_float(bb, eb) * ((ea + eb) & 1 ? 2.0f : 1.0f);
  const float c2v = fr * fr + fi * fi;
  off = c2v > 0.0f ? sqrtf(c2v / ab) : 0.0f;
  R.on = off > (float)tol;
  if (!R.on) return R;
  const int lane = threadIdx.x & 31;
  const float rc = rsqrtf(c2v);
  const double pr = (double)(fr * rc), pi = (double)(-fi * rc);
  const double diff = bb - aa;
  const float z = scaled_float(diff, h) * 0.5f * rc;
  if (!(fabsf(z) < 1e15f)) return rotation_fp64(aa, bb, cr, ci, tol, off);
  const double t = (double)(copysignf(1.0f, z) / (fabsf(z) + sqrtf(1.0f + z * z)));
  const double v = inv_norm(lane == 0 ? t : pr, lane == 0 ? 1.0 : pi);
  R.cs = __shfl_sync(0xffffffffu, v, 0);
  const double s = __shfl_sync(0xffffffffu, v, 1);
  R.sn = R.cs * t;
  const double qr = pr * s, qi = pi * s;
  R.gr = R.sn * qr;
  R.gi = R.sn * qi;
  R.hr = R.cs * qr;
  R.hi = R.cs * qi;
  return R;
}

template <typename T, typename T2>
__device__ __forceinline__ void rotate(const Rot<T>& R, T2& x, T2& y) {
  T2 u, v;
  u.x = R.cs * x.x;
  u.x = fma(-R.gr, y.x, u.x);
  u.x = fma(R.gi, y.y, u.x);
  u.y = R.cs * x.y;
  u.y = fma(-R.gr, y.y, u.y);
  u.y = fma(-R.gi, y.x, u.y);
  v.x = R.sn * x.x;
  v.x = fma(R.hr, y.x, v.x);
  v.x = fma(-R.hi, y.y, v.x);
  v.y = R.sn * x.y;
  v.y = fma(R.hr, y.y, v.y);
  v.y = fma(R.hi, y.x, v.y);
  x = u;
  y = v;
}

__device__ __forceinline__ void group_sync(int g) {
  asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "r"(GROUP) : "memory");
}

// The sweeps over W (p x r) and V (r x r), column-major in global memory, by a cluster;
// returns the number of sweeps. A sweep in which no pair was further from orthogonal than
// `last` is the last one (0: a sweep without rotations is).
template <typename T>
__device__ int sweeps(typename Cplx<T>::type* __restrict__ W, typename Cplx<T>::type* __restrict__ V,
                      int p, int r, T tol, float last, int max_sweeps) {
  typedef typename Cplx<T>::type T2;
  cg::cluster_group cluster = cg::this_cluster();
  const int cs = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = tid & 31;
  const int g = tid / GROUP, gt = tid % GROUP, gw = gt >> 5;
  __shared__ T s_sum[NGROUP][4][4];
  __shared__ Rot<T> s_rot[NGROUP];
  __shared__ int s_off[2];          // largest off-orthogonality of a sweep (float bits)
  if (tid < 2) s_off[tid] = 0;
  const int rr = r + (r & 1);       // an odd count plays against an absent column
  cluster.sync();
  int sweep = 0;
  for (; sweep < max_sweeps; ++sweep) {
    int worst = 0;
    for (int q = 0; q < rr - 1; ++q) {
      for (int t = rank + cs * g; t < rr / 2; t += cs * NGROUP) {
        int j = t == 0 ? 0 : 1 + (q + t) % (rr - 1);
        int k = t == 0 ? 1 + q : 1 + (q + rr - 1 - t) % (rr - 1);
        if (j > k) {
          const int x = j;
          j = k;
          k = x;
        }
        if (k >= r) continue;
        T2* wj = W + (long)j * p;
        T2* wk = W + (long)k * p;
        T2* vj = V + (long)j * r;
        T2* vk = V + (long)k * r;
        T2 x[REG], y[REG], a, b;
        T aa = 0, bb = 0, cr = 0, ci = 0;
#pragma unroll
        for (int e = 0; e < REG; ++e) {
          const int i = gt + e * GROUP;
          if (i < p) {
            x[e] = __ldcg(wj + i);
            y[e] = __ldcg(wk + i);
          } else {
            x[e].x = x[e].y = y[e].x = y[e].y = 0;
          }
        }
        if (gt < r) {
          a = __ldcg(vj + gt);
          b = __ldcg(vk + gt);
        }
        auto gram = [&](const T2& u, const T2& v) {
          aa = fma(u.x, u.x, fma(u.y, u.y, aa));
          bb = fma(v.x, v.x, fma(v.y, v.y, bb));
          cr = fma(u.x, v.x, fma(u.y, v.y, cr));   // conj(u) v
          ci = fma(u.x, v.y, fma(-u.y, v.x, ci));
        };
#pragma unroll
        for (int e = 0; e < REG; ++e)
          if (e * GROUP < p) gram(x[e], y[e]);
        for (int i = gt + REG * GROUP; i < p; i += GROUP) gram(__ldcg(wj + i), __ldcg(wk + i));
        const T sum = warp_sum4(aa, bb, cr, ci);
        if (lane < 4) s_sum[g][gw][lane] = sum;
        group_sync(g);
        if (gw == (g & 3)) {   // one warp per sub-partition forms its group's rotation
          T v = 0;
          if (lane < 4)
            v = (s_sum[g][0][lane] + s_sum[g][1][lane]) + (s_sum[g][2][lane] + s_sum[g][3][lane]);
          float off;
          const Rot<T> R = rotation(__shfl_sync(0xffffffffu, v, 0), __shfl_sync(0xffffffffu, v, 1),
                                    __shfl_sync(0xffffffffu, v, 2), __shfl_sync(0xffffffffu, v, 3),
                                    tol, off);
          if (lane == 0) s_rot[g] = R;
          if (R.on) worst = max(worst, __float_as_int(off));
        }
        group_sync(g);
        const Rot<T> R = s_rot[g];
        if (!R.on) continue;
#pragma unroll
        for (int e = 0; e < REG; ++e) {
          const int i = gt + e * GROUP;
          if (e * GROUP < p) rotate(R, x[e], y[e]);
          if (i < p) {
            __stcg(wj + i, x[e]);
            __stcg(wk + i, y[e]);
          }
        }
        for (int i = gt + REG * GROUP; i < p; i += GROUP) {
          T2 u = __ldcg(wj + i), v = __ldcg(wk + i);
          rotate(R, u, v);
          __stcg(wj + i, u);
          __stcg(wk + i, v);
        }
        if (gt < r) {
          rotate(R, a, b);
          __stcg(vj + gt, a);
          __stcg(vk + gt, b);
        }
        for (int i = gt + GROUP; i < r; i += GROUP) {
          T2 u = __ldcg(vj + i), v = __ldcg(vk + i);
          rotate(R, u, v);
          __stcg(vj + i, u);
          __stcg(vk + i, v);
        }
      }
      cluster.sync();
    }
    // the largest off-orthogonality of the sweep, over the cluster
    if (worst > 0 && lane == 0)
      for (int c = 0; c < cs; ++c) atomicMax(cluster.map_shared_rank(&s_off[sweep & 1], c), worst);
    if (tid == 0) s_off[(sweep + 1) & 1] = 0;
    cluster.sync();
    const float off = __int_as_float(s_off[sweep & 1]);
    if (off <= last) break;
    // everyone has read it before the next but one sweep clears it
  }
  cluster.sync();
  return sweep;
}

// biased exponent of the largest component of A (2047: an infinity or NaN), by the cluster
__device__ int largest_exponent(const double2* __restrict__ a, int m, int n, long lda) {
  cg::cluster_group cluster = cg::this_cluster();
  const int cs = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  __shared__ int s_max;
  if (threadIdx.x == 0) s_max = 0;
  cluster.sync();
  int e = 0;
  for (long q = rank * (long)ST + threadIdx.x; q < (long)m * n; q += (long)cs * ST) {
    const double2 z = a[(q / n) * lda + q % n];
    e = max(e, max((int)((__double_as_longlong(z.x) >> 52) & 0x7FF),
                   (int)((__double_as_longlong(z.y) >> 52) & 0x7FF)));
  }
  e = __reduce_max_sync(0xffffffffu, e);
  if ((threadIdx.x & 31) == 0)
    for (int c = 0; c < cs; ++c) atomicMax(cluster.map_shared_rank(&s_max, c), e);
  cluster.sync();
  return s_max;
}

// Y = I + X from G = W^H W (r x r, row-major), see the top of the file
__global__ void svd_first_order_kernel(const double2* __restrict__ G, int r, double2* __restrict__ Y,
                                       double xmax, const int* __restrict__ bad) {
  if (*bad != 0) return;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < (long)r * r;
       e += (long)gridDim.x * blockDim.x) {
    const int i = (int)(e / r), j = (int)(e % r);
    double2 y = c2(i == j ? 1.0 : 0.0, 0.0);
    if (i != j) {
      // both elements of a pair from the one above the diagonal: G is Hermitian up to rounding
      // only, and where singular values repeat its off-diagonal part is nothing but rounding
      const double2 t = i < j ? G[e] : cconj(G[(long)j * r + i]);
      const double d = G[(long)j * r + j].x - G[(long)i * r + i].x;
      if (fabs(t.x) + fabs(t.y) <= xmax * fabs(d) && d != 0.0) y = c2(t.x / d, t.y / d);
    }
    Y[e] = y;
  }
}

// The FP32 sweeps with the columns of W and V in shared memory, for matrices whose two copies
// fit the cluster (SHARED_MAX a CTA; others stay in L2, above). Pair t of a round lives in CTA
// t / S; in the circle order a pair's first column goes to pair t - 1 for the next round and
// its second to pair t + 1, so a rotation writes its columns where the next round reads them,
// into the other copy, mostly in the same CTA. Every warp forms its group's rotation itself.
// What bounds it: latency of a round (sums over the group, the rotation, the cluster barrier).
// Measured, 128 x 96: 1525 us through L2 -> 956 us (no integer division in a round, approximate
// FP32 divisions and roots in the rotation: 1320 us without these two).
constexpr long SHARED_MAX = 192 * 1024;
constexpr long pre_pairs(long r, long cs) { return ((r + 1) / 2 + cs - 1) / cs; }   // S
constexpr long pre_bytes(long p, long r, long cs) {
  return pre_pairs(r, cs) * 2 * 2 * (p + r) * (long)sizeof(float2);
}

__device__ void sweeps_shared(float2* sh, const double2* __restrict__ a, long lda, bool wide, int p,
                              int r, int ex, float tol, float last, int max_sweeps,
                              double2* __restrict__ Vd) {
  cg::cluster_group cluster = cg::this_cluster();
  const int cs = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = tid & 31;
  const int g = tid / GROUP, gt = tid % GROUP, gw = gt >> 5;
  __shared__ float s_sum[NGROUP][2][4][4];
  __shared__ int s_off[2];
  if (tid < 2) s_off[tid] = 0;
  const int T = (r + 1) / 2, ring = 2 * T - 1;   // pairs, columns in the circle
  const int S = (int)pre_pairs(r, cs), len = p + r;
  const int mine = max(0, min(S, T - rank * S));
  auto first_of = [&](int q, int t) { return t == 0 ? 0 : 1 + (q + t) % ring; };
  auto second_of = [&](int q, int t) { return 1 + (q + ring - t) % ring; };
  for (int e = tid; e < mine * 2 * len; e += ST) {
    const int h = e / len, i = e % len, t = rank * S + (h >> 1);
    const int c = h & 1 ? second_of(0, t) : first_of(0, t);
    float2 v = make_float2(i - p == c ? 1.0f : 0.0f, 0.0f);
    if (i < p && c < r) {   // the column that makes an odd count even is zero
      double2 z = wide ? a[(long)c * lda + i] : a[(long)i * lda + c];
      if (wide) z.y = -z.y;
      v = make_float2(scaled_float(z.x, ex - 1022), scaled_float(z.y, ex - 1022));
    }
    sh[e] = v;
  }
  cluster.sync();
  int b = 0, par = 0;
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    int worst = 0;
    for (int q = 0; q < ring; ++q) {
      for (int s = g; s < mine; s += NGROUP) {
        const int t = rank * S + s;
        const float2* x = sh + (b * S + s) * 2 * len;
        const float2* y = x + len;
        auto place = [&](int by, int side) {   // in pair t + by; no divisions in here
          const int to = s + by, rk = rank + (to < 0 ? -1 : to == S ? 1 : 0);
          const int sl = to < 0 ? S - 1 : to == S ? 0 : to;
          return cluster.map_shared_rank(sh, rk) + ((b ^ 1) * S + sl) * 2 * len + side * len;
        };
        float2* nx = place(t == 0 ? 0 : -1, t == 1 ? 1 : 0);
        float2* ny = t == T - 1 ? place(0, 0) : place(1, 1);
        Rot<float> R;
        R.on = 0;
        if (r == ring + 1 || max(first_of(q, t), second_of(q, t)) < r) {
          float aa = 0.0f, bb = 0.0f, cr = 0.0f, ci = 0.0f;
          for (int i = gt; i < p; i += GROUP) {
            const float2 u = x[i], v = y[i];
            aa = fmaf(u.x, u.x, fmaf(u.y, u.y, aa));
            bb = fmaf(v.x, v.x, fmaf(v.y, v.y, bb));
            cr = fmaf(u.x, v.x, fmaf(u.y, v.y, cr));   // conj(u) v
            ci = fmaf(u.x, v.y, fmaf(-u.y, v.x, ci));
          }
          const float sum = warp_sum4(aa, bb, cr, ci);
          float(*part)[4] = s_sum[g][par];
          par ^= 1;   // a warp may be one pair ahead of the others
          if (lane < 4) part[gw][lane] = sum;
          group_sync(g);
          float v[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) v[k] = (part[0][k] + part[1][k]) + (part[2][k] + part[3][k]);
          float off;
          R = rotation(v[0], v[1], v[2], v[3], tol, off);
          if (R.on) worst = max(worst, __float_as_int(off));
        }
        for (int i = gt; i < len; i += GROUP) {
          float2 u = x[i], v = y[i];
          if (R.on) rotate(R, u, v);
          nx[i] = u;
          ny[i] = v;
        }
      }
      cluster.sync();
      b ^= 1;
    }
    // the largest off-orthogonality of the sweep, over the cluster
    if (worst > 0 && lane == 0)
      for (int c = 0; c < cs; ++c) atomicMax(cluster.map_shared_rank(&s_off[sweep & 1], c), worst);
    if (tid == 0) s_off[(sweep + 1) & 1] = 0;
    cluster.sync();
    if (__int_as_float(s_off[sweep & 1]) <= last) break;
    // everyone has read it before the next but one sweep clears it
  }
  // a whole sweep brings every column back to its first place
  for (int e = tid; e < mine * 2 * r; e += ST) {
    const int h = e / r, i = e % r, t = rank * S + (h >> 1);
    const int c = h & 1 ? second_of(0, t) : first_of(0, t);
    if (c < r) {
      const float2 v = sh[((long)b * S * 2 + h) * len + p + i];
      Vd[(long)c * r + i] = c2(v.x, v.y);
    }
  }
}

// FP32 sweeps on A scaled to entries below 1: V32 as FP64 to Vd (column-major), identities
// to the NS buffers G (for the Newton-Schulz steps), *bad = 1 when A holds an infinity or NaN, or
// entries whose squares would leave the range in the Gram matrices (the GEMMs are skipped and the
// FP64 sweeps start from A itself).
__global__ void __launch_bounds__(ST) svd_pre_kernel(const double2* __restrict__ a, int m, int n,
                                                     long lda, float2* __restrict__ W,
                                                     float2* __restrict__ V,
                                                     double2* __restrict__ Vd,
                                                     double2* __restrict__ G,
                                                     int* __restrict__ bad, bool shared) {
  extern __shared__ float2 columns[];
  cg::cluster_group cluster = cg::this_cluster();
  const int cs = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int tid = threadIdx.x;
  const bool wide = m < n;
  const int p = wide ? n : m, r = wide ? m : n;
  const long step = (long)cs * ST, first = rank * (long)ST + tid;
  const int e = largest_exponent(a, m, n, lda);
  const bool skip = e > 1023 + RANGE;
  if (rank == 0 && tid == 0) *bad = skip ? 1 : 0;
  if (!skip && shared) {
    sweeps_shared(columns, a, lda, wide, p, r, e, 1e-6f, 3e-4f, PRE_SWEEPS, Vd);
  } else if (!skip) {
    for (long q = first; q < (long)p * r; q += step) {
      const int j = (int)(q / p), i = (int)(q % p);
      double2 z = wide ? a[(long)j * lda + i] : a[(long)i * lda + j];
      if (wide) z.y = -z.y;
      __stcg(W + q, make_float2(scaled_float(z.x, e - 1022), scaled_float(z.y, e - 1022)));
    }
    for (long q = first; q < (long)r * r; q += step)
      __stcg(V + q, make_float2(q / r == q % r ? 1.0f : 0.0f, 0.0f));
    cluster.sync();
    sweeps<float>(W, V, p, r, 1e-6f, 3e-4f, PRE_SWEEPS);
  }
  for (long q = first; q < (long)r * r; q += step) {
    const double2 one = c2(q / r == q % r ? 1.0 : 0.0, 0.0);
#pragma unroll
    for (int t = 0; t < NS; ++t) G[(long)t * r * r + q] = one;
    if (!skip && !shared) {
      const float2 v = __ldcg(V + q);
      Vd[q] = c2(v.x, v.y);
    }
  }
  cluster.sync();
}

// whether a pair of the Gram matrix H = W^H W is further from orthogonal than tol, by the
// cluster: the test that a sweep makes pair by pair, with its exceptions (columns near the
// lower end of the range are left to it)
__device__ bool pair_left(const double2* __restrict__ H, int r, float tol) {
  cg::cluster_group cluster = cg::this_cluster();
  const int cs = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  __shared__ int s_left;
  if (threadIdx.x == 0) s_left = 0;
  cluster.sync();
  bool left = false;
  for (long e = rank * (long)ST + threadIdx.x; e < (long)r * r; e += (long)cs * ST) {
    const int i = (int)(e / r), j = (int)(e % r);
    if (i >= j) continue;
    const double2 h = H[e];
    const double aa = H[(long)i * r + i].x, bb = H[(long)j * r + j].x;
    const int ea = exp_of(aa), eb = exp_of(bb), sh = (ea + eb) >> 1;
    if (ea == 1024 || eb == 1024) continue;
    const float fr = scaled_float(h.x, sh), fi = scaled_float(h.y, sh);
    const float ab = scaled_float(aa, ea) * scaled_float(bb, eb) * ((ea + eb) & 1 ? 2.0f : 1.0f);
    left |= ea < -960 || eb < -960 || !(fr * fr + fi * fi <= tol * tol * ab);
  }
  if (__any_sync(0xffffffffu, left) && (threadIdx.x & 31) == 0)
    for (int c = 0; c < cs; ++c) *cluster.map_shared_rank(&s_left, c) = 1;
  cluster.sync();
  return s_left != 0;
}

// W (p x r) and V (r x r) are column-major scratch; u, vh row-major outputs. `pre`: W and V
// hold the start of the sweeps unless *bad.
__global__ void __launch_bounds__(ST) svd_jacobi_kernel(const double2* __restrict__ a, int m, int n,
                                                       long lda, double2* __restrict__ W,
                                                       double2* __restrict__ V,
                                                       double* __restrict__ sig,
                                                       int* __restrict__ pos, double2* __restrict__ u,
                                                       long ldu, double* __restrict__ s,
                                                       double2* __restrict__ vh, long ldvh,
                                                       int* __restrict__ sweeps_out, int pre,
                                                       const int* __restrict__ bad,
                                                       const double2* __restrict__ H) {
  cg::cluster_group cluster = cg::this_cluster();
  const int cs = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = rank * (ST / 32) + (tid >> 5), nwarp = cs * (ST / 32);
  const bool wide = m < n;
  const int p = wide ? n : m, r = wide ? m : n;
  const long step = (long)cs * ST, first = rank * (long)ST + tid;
  // entries whose squares would leave the FP64 range: W carries a power of two
  const int ea = largest_exponent(a, m, n, lda);
  const int shift = (ea != 0 && ea != 2047 && abs(ea - 1023) > RANGE) ? 1023 - ea : 0;
  if (!pre || *bad != 0) {
    for (long e = first; e < (long)p * r; e += step) {
      const int j = (int)(e / p), i = (int)(e % p);
      double2 z = wide ? cconj(a[(long)j * lda + i]) : a[(long)i * lda + j];
      if (shift != 0) z = c2(ldexp(z.x, shift), ldexp(z.y, shift));
      __stcg(W + e, z);
    }
    for (long e = first; e < (long)r * r; e += step)
      __stcg(V + e, c2((e / r == e % r) ? 1.0 : 0.0, 0.0));
  } else if (shift != 0) {
    for (long e = first; e < (long)p * r; e += step)
      __stcg(W + e, c2(ldexp(W[e].x, shift), ldexp(W[e].y, shift)));
  }
  cluster.sync();
  const double tol = (double)p * 2.220446049250313e-16;
  int sweep = 0;
  if (!pre || *bad != 0 || shift != 0 || pair_left(H, r, (float)tol))
    sweep = sweeps<double>(W, V, p, r, tol, 0.0f, MAX_SWEEPS);
  // singular values, their order, the outputs
  for (int j = warp; j < r; j += nwarp) {
    const double2* wj = W + (long)j * p;
    double acc = 0.0;
    for (int i = lane; i < p; i += 32) {
      const double2 z = __ldcg(wj + i);
      acc = fma(z.x, z.x, fma(z.y, z.y, acc));
    }
    acc = warp_sum(acc);
    if (lane == 0) __stcg(sig + j, sqrt(acc));
  }
  cluster.sync();
  for (int j = (int)first; j < r; j += (int)step) {
    const double sj = __ldcg(sig + j);
    int c = 0;
    for (int i = 0; i < r; ++i) {
      const double si = __ldcg(sig + i);
      c += (si > sj || (si == sj && i < j)) ? 1 : 0;
    }
    __stcg(pos + j, c);
    s[c] = shift != 0 ? ldexp(sj, -shift) : sj;
  }
  cluster.sync();
  // tall: U[i][pos j] = w_j[i] / s_j, Vh[pos j][c] = conj(V[c][j]); wide: A^H = U_w diag(s)
  // V^H, so U[i][pos j] = V[i][j], Vh[pos j][c] = conj(w_j[c]) / s_j. One warp per column.
  for (int j = warp; j < r; j += nwarp) {
    const double sj = __ldcg(sig + j);
    const int c = __ldcg(pos + j);
    const double inv = sj > 0.0 ? 1.0 / sj : 0.0;
    for (int i = lane; i < p; i += 32) {
      const double2 x = __ldcg(W + (long)j * p + i);
      if (!wide) u[(long)i * ldu + c] = c2(x.x * inv, x.y * inv);
      else vh[(long)c * ldvh + i] = c2(x.x * inv, -x.y * inv);
    }
    for (int i = lane; i < r; i += 32) {
      const double2 x = __ldcg(V + (long)j * r + i);
      if (!wide) vh[(long)c * ldvh + i] = cconj(x);
      else u[(long)i * ldu + c] = x;
    }
  }
  if (rank == 0 && tid == 0 && sweeps_out != nullptr)
    *sweeps_out = sweep + (sweep == MAX_SWEEPS ? 1 : 0);
}

// a[i][j] *= s[j] (side 0: columns) or s[i] (side 1: rows), row-major with ld
__global__ void diag_scale_kernel(double2* __restrict__ a, long rows, long cols, long ld,
                                  const double* __restrict__ s, int side) {
  const long total = rows * cols;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total;
       e += (long)gridDim.x * blockDim.x) {
    const long i = e / cols, j = e % cols;
    const double f = s[side == 0 ? j : i];
    double2* x = a + i * ld + j;
    *x = c2(x->x * f, x->y * f);
  }
}

inline size_t al(size_t b) { return (b + 255) & ~size_t(255); }

}  // namespace

// largest cluster the kernels can be launched with (16, else 8, else 1); decided once
// and whether the FP32 kernel fits with its columns in shared memory
static int svd_cluster_max(bool* shared = nullptr) {
  static int best = 1;
  static bool fits = false;
  static std::once_flag once;
  std::call_once(once, [] {
    for (const void* f : {(const void*)svd_pre_kernel, (const void*)svd_jacobi_kernel})
      if (cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
        cudaGetLastError();
    for (int c : {16, 8}) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(c);
      cfg.blockDim = dim3(ST);
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = c;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      int na = 0, nb = 0;
      if (cudaOccupancyMaxActiveClusters(&na, svd_pre_kernel, &cfg) == cudaSuccess &&
          cudaOccupancyMaxActiveClusters(&nb, svd_jacobi_kernel, &cfg) == cudaSuccess && na > 0 &&
          nb > 0) {
        best = c;
        if (cudaFuncSetAttribute(svd_pre_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)SHARED_MAX) == cudaSuccess) {
          cfg.dynamicSmemBytes = SHARED_MAX;
          fits = cudaOccupancyMaxActiveClusters(&na, svd_pre_kernel, &cfg) == cudaSuccess && na > 0;
        }
        if (!fits) cudaGetLastError();
        break;
      }
      cudaGetLastError();
    }
  });
  if (shared != nullptr) *shared = fits;
  return best;
}

struct SvdWs {
  double2 *W, *V;
  double* sig;
  int *pos, *bad;
  // FP32 start
  float2 *W32, *V32;
  double2 *V0, *G, *H, *Y;   // V's second buffer, NS identities, W^H W, I + X
};

static size_t svd_layout(void* base, long p, long r, SvdWs* w) {
  size_t off = 0;
  auto take = [&](size_t bytes) {
    void* q = base ? static_cast<char*>(base) + off : nullptr;
    off += al(bytes);
    return q;
  };
  w->W = static_cast<double2*>(take((size_t)p * r * sizeof(double2)));
  w->V = static_cast<double2*>(take((size_t)r * r * sizeof(double2)));
  w->sig = static_cast<double*>(take((size_t)r * sizeof(double)));
  w->pos = static_cast<int*>(take((size_t)(r + 1) * sizeof(int)));
  w->bad = w->pos ? w->pos + r : nullptr;
  if (r >= PRE_MIN) {
    w->W32 = static_cast<float2*>(take((size_t)p * r * sizeof(float2)));
    w->V32 = static_cast<float2*>(take((size_t)r * r * sizeof(float2)));
    w->V0 = static_cast<double2*>(take((size_t)r * r * sizeof(double2)));
    w->G = static_cast<double2*>(take((size_t)NS * r * r * sizeof(double2)));
    w->H = static_cast<double2*>(take((size_t)r * r * sizeof(double2)));
    w->Y = static_cast<double2*>(take((size_t)r * r * sizeof(double2)));
  }
  return off;
}

size_t svd_workspace_bytes(int m, int n) {
  SvdWs w;
  return svd_layout(nullptr, std::max(m, n), std::min(m, n), &w);
}

ptn_status svd(const double2* a, int m, int n, long lda, double2* u, long ldu, double* s,
               double2* vh, long ldvh, int* sweeps, void* ws, size_t ws_bytes, cudaStream_t st) {
  PTN_CHECK_ARG(m > 0 && n > 0, "svd: empty matrix (%d x %d)", m, n);
  PTN_CHECK_ARG(lda >= n && ldu >= std::min(m, n) && ldvh >= n, "svd: bad leading dimensions");
  PTN_CHECK_ARG(ws_bytes >= svd_workspace_bytes(m, n), "svd: workspace too small");
  const int p = std::max(m, n), r = std::min(m, n);
  const bool wide = m < n, pre = r >= PRE_MIN;
  SvdWs w;
  svd_layout(ws, p, r, &w);
  // one pair per CTA while the cluster allows
  int cs = 1;
  while (cs < svd_cluster_max() && cs < (r + 1) / 2) cs *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cs);
  cfg.blockDim = dim3(ST);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (pre) {
    bool shared = false;
    svd_cluster_max(&shared);
    shared = shared && pre_bytes(p, r, cs) <= SHARED_MAX;
    cfg.dynamicSmemBytes = shared ? pre_bytes(p, r, cs) : 0;
    PTN_CUDA_TRY(cudaLaunchKernelEx(&cfg, svd_pre_kernel, a, m, n, lda, w.W32, w.V32, w.V0, w.G,
                                    w.bad, shared));
    cfg.dynamicSmemBytes = 0;
    note_launches(1);
    // the buffers hold V^T and W^T row-major (V and W column by column)
    double2* V = w.V0;
    double2* V2 = w.V;
    auto mult = [&](char oa, char ob, int M, int N, int K, const double2* A, long la,
                    const double2* B, long lb, double2* C, double al, double be) {
      GemmArgs g;
      g.M = M; g.N = N; g.K = K; g.opA = oa; g.opB = ob;
      g.alpha = make_double2(al, 0.0); g.beta = make_double2(be, 0.0);
      g.A = A; g.lda = la; g.sA = 0;
      g.B = B; g.ldb = lb; g.sB = 0;
      g.C = C; g.ldc = N; g.sC = 0;
      g.batch = 1; g.skip = w.bad;
      return zgemm(g, nullptr, 0, st);
    };
    auto newton_schulz = [&](int t) -> ptn_status {   // V <- V (3 I - V^H V) / 2
      double2* G = w.G + (long)t * r * r;
      PTN_TRY(mult('C', 'T', r, r, r, V, r, V, r, G, -0.5, 1.5));
      PTN_TRY(mult('T', 'N', r, r, r, G, r, V, r, V2, 1.0, 0.0));
      std::swap(V, V2);
      return PTN_OK;
    };
    auto times_a = [&]() {   // W = A V (tall) or A^H V (wide)
      return mult('N', wide ? 'C' : 'T', r, p, r, V, r, a, lda, w.W, 1.0, 0.0);
    };
    PTN_TRY(newton_schulz(0));
    PTN_TRY(times_a());
    for (int t = 0; t < REFINE; ++t) {
      PTN_TRY(mult('C', 'T', r, r, p, w.W, p, w.W, p, w.H, 1.0, 0.0));
      svd_first_order_kernel<<<std::min(4 * num_sms(), (r * r + 127) / 128), 128, 0, st>>>(
          w.H, r, w.Y, X_NORM[t] / r, w.bad);
      PTN_LAUNCH_CHECK();
      note_launches(1);
      PTN_TRY(mult('T', 'N', r, r, r, w.Y, r, V, r, V2, 1.0, 0.0));   // V (I + X)
      std::swap(V, V2);
      PTN_TRY(newton_schulz(2 * t + 1));
      PTN_TRY(newton_schulz(2 * t + 2));
      PTN_TRY(times_a());
    }
    PTN_TRY(mult('C', 'T', r, r, p, w.W, p, w.W, p, w.H, 1.0, 0.0));   // for the last check
    w.V = V;
  }
  PTN_CUDA_TRY(cudaLaunchKernelEx(&cfg, svd_jacobi_kernel, a, m, n, lda, w.W, w.V, w.sig, w.pos, u,
                                  ldu, s, vh, ldvh, sweeps, pre ? 1 : 0, (const int*)w.bad, (const double2*)w.H));
  PTN_LAUNCH_CHECK();
  note_launches(1);
  return PTN_OK;
}

}  // namespace ptn

extern "C" {

size_t ptn_svd_workspace_bytes(int m, int n) { return ptn::svd_workspace_bytes(m, n); }

ptn_status ptn_svd(const ptn_c128* a, int m, int n, long lda, ptn_c128* u, long ldu, double* s,
                   ptn_c128* vh, long ldvh, int* sweeps, void* ws, size_t ws_bytes,
                   void* stream) {
  return ptn::svd(reinterpret_cast<const double2*>(a), m, n, lda, reinterpret_cast<double2*>(u),
                  ldu, s, reinterpret_cast<double2*>(vh), ldvh, sweeps, ws, ws_bytes,
                  ptn::as_stream(stream));
}

ptn_status ptn_diag_scale(ptn_c128* a, long rows, long cols, long ld, const double* s, int side,
                          void* stream) {
  PTN_CHECK_ARG(rows >= 0 && cols >= 0 && ld >= cols && (side == 0 || side == 1),
                "diag_scale: bad arguments");
  if (rows == 0 || cols == 0) return PTN_OK;
  cudaStream_t st = ptn::as_stream(stream);
  const long total = rows * cols;
  const int blocks = (int)std::max(1L, std::min((total + 255) / 256, 8L * ptn::num_sms()));
  ptn::diag_scale_kernel<<<blocks, 256, 0, st>>>(reinterpret_cast<double2*>(a), rows, cols, ld,
                                                 s, side);
  PTN_LAUNCH_CHECK();
  ptn::note_launches(1);
  return PTN_OK;
}

}  // extern "C"
