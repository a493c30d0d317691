// Complex128 GEMM on the FP64 DMMA tensor-core path (mma.sync m8n8k4 f64).
//
// C = alpha op(A) op(B) + beta C, all row-major, op in {N, T, C, H}. This is the
// contraction engine of the plain (all-FP64) form: every tensordot of
// pytenet/chain_ops.py (apply_local_hamiltonian, the environment steps, the bond
// contraction) and of the sweep (pytenet/tdvp.py:84,112) becomes one call.
//
// What bounds it: an SM executes two FP64 FMAs per cycle whatever the instruction, so a
// DMMA (256 FMAs) occupies its sub-partition for 512 cycles and the four DMMAs of a
// complex 8 x 8 x 4 step for 2048. Next to that the operands cost nothing (1 KB per
// step), so nothing is staged through shared memory: a warp owns one 8 x 8 block of C
// and loads its fragments straight from L2 / L1 into registers, two steps ahead. What
// matters is that no sub-partition multiplies padding or idles: the unit of work is one
// warp's block (not a 64 x 64 tile), and blocks that are too few for the chip's 608
// sub-partitions split K over the four warps of a CTA and over the CTAs of a cluster,
// summed through (distributed) shared memory in a fixed order: no partial sums in
// global memory, no second launch.
// Measured against the 64 x 64 x 16 shared-memory tiles this replaces (one call of
// H_eff . A, its two GEMMs): see choose_shape.
// Transposition and conjugation are folded into the loads.
//
// Block sparsity: a K step whose A fragment (8 x 4) or B fragment (4 x 8) is entirely
// zero contributes nothing and its DMMAs are skipped (a warp vote; not when the other
// fragment holds an infinity or NaN, whose product with zero is NaN). Tensors with
// quantum numbers hold zero blocks (pytenet/block_sparse_util.py:47-64), which after
// the first block QR line up with these fragments.
#include "ptn_common.cuh"
#include "launch.cuh"
#include "rns.cuh"
#include <cooperative_groups.h>
#include <algorithm>
#include <cmath>

namespace cg = cooperative_groups;

namespace ptn {
namespace {

constexpr int FB = 8;              // rows and columns of a warp's block
constexpr int WARPS = 4;
constexpr int THREADS = 32 * WARPS;
constexpr int MAX_CLUSTER = 8;

enum { OP_N = 0, OP_T = 1, OP_C = 2, OP_H = 3 };

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

template <int OP>
struct OpTraits {
  static constexpr bool trans = (OP == OP_T || OP == OP_H);
  static constexpr bool conj = (OP == OP_C || OP == OP_H);
};

struct KArgs {
  int M, N, K;
  int kchunk;                       // K entries per part (a multiple of 4)
  double2 alpha, beta;
  const double2* A; long lda, sA;
  const double2* B; long ldb, sB;
  double2* C; long ldc, sC;
  const int* skip;
};

// op(X)[r][k] of a fragment lane, zero outside
template <int OP>
__device__ __forceinline__ double2 frag_a(const double2* __restrict__ A, long lda, int r, int k,
                                          int M, int kend) {
  double2 v = make_double2(0.0, 0.0);
  if (r < M && k < kend) v = OpTraits<OP>::trans ? A[(long)k * lda + r] : A[(long)r * lda + k];
  if (OpTraits<OP>::conj) v.y = -v.y;
  return v;
}

template <int OP>
__device__ __forceinline__ double2 frag_b(const double2* __restrict__ B, long ldb, int c, int k,
                                          int N, int kend) {
  double2 v = make_double2(0.0, 0.0);
  if (c < N && k < kend) v = OpTraits<OP>::trans ? B[(long)c * ldb + k] : B[(long)k * ldb + c];
  if (OpTraits<OP>::conj) v.y = -v.y;
  return v;
}

// 1: has a non-zero entry; 2: has an infinity or NaN
__device__ __forceinline__ unsigned entry_class(double2 v) {
  const unsigned hx = (unsigned)__double2hiint(v.x) & 0x7FF00000u;
  const unsigned hy = (unsigned)__double2hiint(v.y) & 0x7FF00000u;
  return ((v.x != 0.0 || v.y != 0.0) ? 1u : 0u) |
         ((hx == 0x7FF00000u || hy == 0x7FF00000u) ? 2u : 0u);
}

// KW = 1: the CTA's four warps own a 2 x 2 group of blocks; KW = 4: they share one
// block, a quarter of the K part each. gridDim.y (= the cluster's y extent) splits K too.
template <int OA, int OB, int KW>
__global__ void __launch_bounds__(THREADS) zgemm_dmma_kernel(const KArgs p) {
  grid_wait();
  if (p.skip != nullptr && *p.skip != 0) return;   // uniform over the launch
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int fr = lane >> 2, fc = lane & 3;
  const int parts = gridDim.y, part = blockIdx.y;
  constexpr int CB = KW == 1 ? 2 * FB : FB;        // CTA block edge
  const int nct = (p.N + CB - 1) / CB;
  const int m0 = (int)(blockIdx.x / nct) * CB + (KW == 1 ? (warp >> 1) * FB : 0);
  const int n0 = (int)(blockIdx.x % nct) * CB + (KW == 1 ? (warp & 1) * FB : 0);
  const double2* A = p.A + (long)blockIdx.z * p.sA;
  const double2* B = p.B + (long)blockIdx.z * p.sB;
  const int kp = (KW == 1) ? part : part * KW + warp;
  const int kbeg = kp * p.kchunk;
  const int kend = min(p.K, kbeg + p.kchunk);
  const int r = m0 + fr, c = n0 + fr;

  double re[2] = {0.0, 0.0}, im[2] = {0.0, 0.0};
  if (m0 < p.M && n0 < p.N && kbeg < kend) {
    double2 a0 = frag_a<OA>(A, p.lda, r, kbeg + fc, p.M, kend);
    double2 b0 = frag_b<OB>(B, p.ldb, c, kbeg + fc, p.N, kend);
    double2 a1 = frag_a<OA>(A, p.lda, r, kbeg + 4 + fc, p.M, kend);
    double2 b1 = frag_b<OB>(B, p.ldb, c, kbeg + 4 + fc, p.N, kend);
    for (int k = kbeg; k < kend; k += 4) {
      const double2 a = a0, b = b0;
      a0 = a1;
      b0 = b1;
      a1 = frag_a<OA>(A, p.lda, r, k + 8 + fc, p.M, kend);
      b1 = frag_b<OB>(B, p.ldb, c, k + 8 + fc, p.N, kend);
      const unsigned ca = entry_class(a), cb = entry_class(b);
      const bool za = !__any_sync(0xffffffffu, ca & 1u), zb = !__any_sync(0xffffffffu, cb & 1u);
      if ((za || zb) && !__any_sync(0xffffffffu, (ca | cb) & 2u)) continue;
      dmma(re[0], re[1], a.x, b.x);
      dmma(im[0], im[1], a.x, b.y);
      dmma(re[0], re[1], -a.y, b.y);
      dmma(im[0], im[1], a.y, b.x);
    }
  }

  // sum the K parts in a fixed order: the warps' quarters, then the cluster's CTAs
  __shared__ double2 s_part[WARPS][2 * 32];
  if (KW == 1 && parts == 1) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int gm = m0 + fr, gn = n0 + 2 * fc + e;
      if (gm < p.M && gn < p.N) {
        double2* cp = p.C + (long)blockIdx.z * p.sC + (long)gm * p.ldc + gn;
        double2 out = cmul(p.alpha, make_double2(re[e], im[e]));
        if (p.beta.x != 0.0 || p.beta.y != 0.0) out = cadd(out, cmul(p.beta, *cp));
        *cp = out;
      }
    }
    return;
  }
  s_part[warp][2 * lane] = make_double2(re[0], im[0]);
  s_part[warp][2 * lane + 1] = make_double2(re[1], im[1]);
  if (parts > 1) cg::this_cluster().sync();
  else __syncthreads();
  // entries of the CTA's blocks, spread over the cluster's CTAs
  constexpr int ENT = (KW == 1 ? WARPS : 1) * 64;
  for (int e = part * THREADS + (int)threadIdx.x; e < ENT; e += parts * THREADS) {
    const int wb = e >> 6, x = e & 63;             // block of the CTA, entry of the block
    double2 s = make_double2(0.0, 0.0);
    for (int q = 0; q < parts; ++q) {
#pragma unroll
      for (int w = 0; w < KW; ++w) {
        const double2* src = &s_part[KW == 1 ? wb : w][x];
        const double2 v = parts > 1 ? *cg::this_cluster().map_shared_rank(src, q) : *src;
        s = (q == 0 && w == 0) ? v : cadd(s, v);
      }
    }
    const int bm = (int)(blockIdx.x / nct) * CB + (wb >> 1) * FB;
    const int bn = (int)(blockIdx.x % nct) * CB + (wb & 1) * FB;
    const int gm = bm + (x >> 3), gn = bn + (x & 7);
    if (gm < p.M && gn < p.N) {
      double2* cp = p.C + (long)blockIdx.z * p.sC + (long)gm * p.ldc + gn;
      double2 out = cmul(p.alpha, s);
      if (p.beta.x != 0.0 || p.beta.y != 0.0) out = cadd(out, cmul(p.beta, *cp));
      *cp = out;
    }
  }
  if (parts > 1) cg::this_cluster().sync();   // no CTA leaves while its shared memory is read
}

int op_code(char c) {
  switch (c) {
    case 'N': case 'n': return OP_N;
    case 'T': case 't': return OP_T;
    case 'C': case 'c': return OP_C;
    case 'H': case 'h': return OP_H;
    default: return -1;
  }
}

struct Shape {
  int kw;       // K parts inside a CTA (1: four blocks per CTA, 4: one)
  int parts;    // CTAs of a cluster that split K
  int kchunk;   // K entries per part
};

// Launch shape: the split of K that finishes first under a plain model: 2048 cycles per
// K step of a block and one block per sub-partition at a time (counted in whole turns
// while there are few), plus what a CTA's and a cluster's sum cost. Measured on the two
// GEMMs of H_eff . A (64 x 64 x 16 tiles with split K through global memory before):
//   bonds 250 x 256, chi 5   1207 + 1485 us -> 1201 + 1423 us (1.01 TF/s)
//   bonds <= 28 (README run)   83 +  213 us ->    4 +    5 us, mean over a time step
//   bonds <= 24, U(1) (DMRG)   87 +  289 us ->    4 +    5 us, mean over a sweep
// PTN_TUNE_ZGEMM_SPLIT_WAVES 0 keeps K within a CTA where it has 128 entries or more; shorter
// products are summed the same way whatever the knob.
Shape choose_shape(int M, int N, int K, int batch) {
  const long subp = 4L * num_sms();
  const long steps = std::max(1, (K + 3) / 4);
  const bool clusters = tune(PTN_TUNE_ZGEMM_SPLIT_WAVES) != 0 || K < 128;
  Shape best{1, 1, 0};
  double best_cost = -1.0;
  for (int kw : {1, 4})
    for (int parts = 1; parts <= (clusters ? MAX_CLUSTER : 1); parts *= 2) {
      const long np = (long)kw * parts;
      if (np > 1 && steps < np) continue;
      const long per = (steps + np - 1) / np;
      const long edge = kw == 1 ? 2 * FB : FB;
      const long ctas = ((M + edge - 1) / edge) * ((N + edge - 1) / edge) * (long)batch * parts;
      const double turns = (double)ctas * WARPS / subp;
      const double whole = turns < 8.0 ? std::ceil(turns) : turns;
      const double cost = whole * (per * 2048.0 + (kw > 1 ? 300.0 : 0.0) + (parts > 1 ? 1200.0 : 0.0));
      if (best_cost < 0.0 || cost < best_cost) {
        best_cost = cost;
        best = Shape{kw, parts, 0};
      }
    }
  const long np = (long)best.kw * best.parts;
  best.kchunk = (int)((steps + np - 1) / np * 4);
  return best;
}

template <int OA, int OB>
cudaError_t launch_ab(const Shape& s, const KArgs& k, int batch, cudaStream_t st) {
  const long edge = s.kw == 1 ? 2 * FB : FB;
  LaunchShape shape{dim3((unsigned)(((k.M + edge - 1) / edge) * ((k.N + edge - 1) / edge)),
                         (unsigned)s.parts, (unsigned)batch), dim3(THREADS), 0};
  if (s.parts > 1) shape.cluster = dim3(1, (unsigned)s.parts, 1);
  if (s.kw == 1) return launch_shape(zgemm_dmma_kernel<OA, OB, 1>, shape, st, k);
  return launch_shape(zgemm_dmma_kernel<OA, OB, 4>, shape, st, k);
}

template <int OA>
cudaError_t launch_b(int ob, const Shape& s, const KArgs& k, int batch, cudaStream_t st) {
  switch (ob) {
    case OP_N: return launch_ab<OA, OP_N>(s, k, batch, st);
    case OP_T: return launch_ab<OA, OP_T>(s, k, batch, st);
    case OP_C: return launch_ab<OA, OP_C>(s, k, batch, st);
    default: return launch_ab<OA, OP_H>(s, k, batch, st);
  }
}

}  // namespace

void note_launches(int n);

// the DMMA kernel splits K inside the launch (clusters) and needs no scratch
size_t zgemm_workspace_bytes(int M, int N, int K, int batch) {
  return batch == 1 && rns_wanted(M, N, K) ? zgemm_rns_workspace_bytes(RNS_FP64, M, N, K) : 0;
}

ptn_status zgemm(const GemmArgs& g, void* ws, size_t ws_bytes, cudaStream_t st) {
  const int oa = op_code(g.opA), ob = op_code(g.opB);
  PTN_CHECK_ARG(oa >= 0 && ob >= 0, "zgemm: bad op (%c, %c)", g.opA, g.opB);
  PTN_CHECK_ARG(g.M >= 0 && g.N >= 0 && g.K >= 0 && g.batch >= 1, "zgemm: bad sizes");
  if (g.M == 0 || g.N == 0) return PTN_OK;
  // a smaller workspace than the query asks for: the DMMA kernel
  if (g.batch == 1 && rns_wanted(g.M, g.N, g.K) && ws != nullptr &&
      ws_bytes >= zgemm_rns_workspace_bytes(RNS_FP64, g.M, g.N, g.K))
    return zgemm_rns(RNS_FP64, g, ws, st);
  KArgs k;
  k.M = g.M; k.N = g.N; k.K = g.K;
  k.alpha = g.alpha; k.beta = g.beta;
  k.A = g.A; k.lda = g.lda; k.sA = g.sA;
  k.B = g.B; k.ldb = g.ldb; k.sB = g.sB;
  k.C = g.C; k.ldc = g.ldc; k.sC = g.sC;
  k.skip = g.skip;
  const Shape s = choose_shape(g.M, g.N, g.K, g.batch);
  k.kchunk = s.kchunk;
  PTN_CHECK_ARG(g.batch <= 65535, "zgemm: grid too large");
  const int prof = prof_begin(st, PROF_ZGEMM_F64, 8.0 * g.M * g.N * (double)g.K * g.batch,
                              16.0 * g.batch * ((double)g.M * g.K + (double)g.K * g.N + 2.0 * g.M * g.N));
  cudaError_t e;
  switch (oa) {
    case OP_N: e = launch_b<OP_N>(ob, s, k, g.batch, st); break;
    case OP_T: e = launch_b<OP_T>(ob, s, k, g.batch, st); break;
    case OP_C: e = launch_b<OP_C>(ob, s, k, g.batch, st); break;
    default: e = launch_b<OP_H>(ob, s, k, g.batch, st); break;
  }
  PTN_CUDA_TRY(e);
  note_launches(1);
  prof_end(st, prof);
  return PTN_OK;
}

}  // namespace ptn

extern "C" {

size_t ptn_zgemm_workspace_bytes(int M, int N, int K, int batch) {
  return ptn::zgemm_workspace_bytes(M, N, K, batch);
}

ptn_status ptn_zgemm(char opA, char opB, int M, int N, int K, ptn_c128 alpha, const ptn_c128* A,
                     long lda, long strideA, const ptn_c128* B, long ldb, long strideB,
                     ptn_c128 beta, ptn_c128* C, long ldc, long strideC, int batch, void* ws,
                     size_t ws_bytes, void* stream) {
  ptn::GemmArgs g;
  g.M = M; g.N = N; g.K = K; g.opA = opA; g.opB = opB;
  g.alpha = make_double2(alpha.re, alpha.im);
  g.beta = make_double2(beta.re, beta.im);
  g.A = reinterpret_cast<const double2*>(A); g.lda = lda; g.sA = strideA;
  g.B = reinterpret_cast<const double2*>(B); g.ldb = ldb; g.sB = strideB;
  g.C = reinterpret_cast<double2*>(C); g.ldc = ldc; g.sC = strideC;
  g.batch = batch; g.skip = nullptr;
  return ptn::zgemm(g, ws, ws_bytes, ptn::as_stream(stream));
}

}  // extern "C"
