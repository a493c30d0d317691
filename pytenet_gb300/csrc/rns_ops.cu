// Site / bond operators and environment steps (pytenet/chain_ops.py:16-99, 237-317) with both
// GEMMs of every contraction in the residue number system (rns.cu): the FP64 form where the
// problem is large enough for it (contract.cu decides), the mixed form nearly always.
//
// Data flow of H_eff . x (site tensors (Dl, d, Dr), MPO bonds cl / cr); an operand is a set
// of residue planes, rows x terms:
//   prepare (once per local step):  R -> rows (wr, r2), terms r0;  L -> rows l2, terms (l0, wl)
//   apply:  x -> rows (l0, t), terms r0
//           GEMM 1 T1[(l0,t)][(wr,r2)], reconstructed inside the MPO stage, which writes
//           T2[l0,(wl,s),r2] in FP64 with the exponents of its rows as the next operand
//           T2 -> rows (s, r2), terms (l0, wl)
//           GEMM 2 out[l2][(s,r2)]
// six launches per apply.
#include "ptn_common.cuh"
#include "rns.cuh"
#include <algorithm>

namespace ptn {

namespace {

constexpr double2 ONE{1.0, 0.0}, ZERO{0.0, 0.0};

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
  RnsOperand operand(long rows, long kc, int nm) {
    void* p = take(rns_plane_bytes(rows, kc, nm));
    void* e = take((size_t)rows * sizeof(int));
    return rns_operand(p, e, rows, kc, nm);
  }
};

#define RNS_CHECK_WS(layout)                                                     \
  do {                                                                           \
    Carver _q(nullptr);                                                          \
    (void)layout(_q);                                                            \
    PTN_CHECK_ARG(ws_bytes >= _q.off, "contraction: workspace too small");       \
  } while (0)

struct HeffWs {
  RnsOperand r, l, x, t2;
  double2* T2;
  void* res;
};

HeffWs heff_ws(Carver& c, int nm, int Dl, int d, int Dr, int cl, int cr) {
  HeffWs w;
  w.r = c.operand((long)cr * Dr, Dr, nm);
  w.l = c.operand(Dl, (long)Dl * cl, nm);
  w.x = c.operand((long)Dl * d, Dr, nm);
  w.t2 = c.operand((long)d * Dr, (long)Dl * cl, nm);
  w.T2 = static_cast<double2*>(c.take((size_t)Dl * cl * d * Dr * sizeof(double2)));
  w.res = c.take(std::max(rns_out_bytes((long)Dl * d, (long)cr * Dr, nm),
                          rns_out_bytes(Dl, (long)d * Dr, nm)));
  return w;
}

struct BondWs {
  RnsOperand r, l, x, t1;
  double2* T1;
  void* res;
};

BondWs bond_ws(Carver& c, int nm, int Dl, int Dr, int chi) {
  BondWs w;
  w.r = c.operand((long)chi * Dr, Dr, nm);
  w.l = c.operand(Dl, (long)Dl * chi, nm);
  w.x = c.operand(Dl, Dr, nm);
  w.t1 = c.operand(Dr, (long)Dl * chi, nm);
  w.T1 = static_cast<double2*>(c.take((size_t)Dl * chi * Dr * sizeof(double2)));
  w.res = c.take(std::max(rns_out_bytes(Dl, (long)chi * Dr, nm), rns_out_bytes(Dl, Dr, nm)));
  return w;
}

// a1 b1: first GEMM, a2 b2: second one
struct EnvWs {
  RnsOperand a1, b1, a2, b2;
  double2* T2;
  void* res;
};

EnvWs env_left_ws(Carver& c, int nm, int Dl, int d, int Dr, int cl, int cr) {
  EnvWs w;
  w.a1 = c.operand((long)Dl * cl, Dl, nm);             // L, rows (l0, wl), terms l2
  w.b1 = c.operand((long)d * Dr, Dl, nm);              // conj(B), rows (t, rb), terms l2
  w.a2 = c.operand(Dr, (long)Dl * d, nm);              // A, rows ra, terms (l0, s)
  w.b2 = c.operand((long)cr * Dr, (long)Dl * d, nm);   // T2, rows (wr, rb), terms (l0, s)
  w.T2 = static_cast<double2*>(c.take((size_t)Dl * d * cr * Dr * sizeof(double2)));
  w.res = c.take(std::max(rns_out_bytes((long)Dl * cl, (long)d * Dr, nm),
                          rns_out_bytes(Dr, (long)cr * Dr, nm)));
  return w;
}

EnvWs env_right_ws(Carver& c, int nm, int Dl, int d, int Dr, int cl, int cr) {
  EnvWs w;
  w.a1 = c.operand((long)Dl * d, Dr, nm);              // A, rows (l0, s), terms r0
  w.b1 = c.operand((long)cr * Dr, Dr, nm);             // R, rows (wr, r2), terms r0
  w.a2 = c.operand((long)Dl * cl, (long)d * Dr, nm);   // T2, rows (l0, wl), terms (t, r2)
  w.b2 = c.operand(Dl, (long)d * Dr, nm);              // conj(B), rows lb, terms (t, r2)
  w.T2 = static_cast<double2*>(c.take((size_t)Dl * cl * d * Dr * sizeof(double2)));
  w.res = c.take(std::max(rns_out_bytes((long)Dl * d, (long)cr * Dr, nm),
                          rns_out_bytes((long)Dl * cl, Dl, nm)));
  return w;
}

}  // namespace

// ================================================================ site operator
size_t heff_workspace_bytes_rns(int nm, int Dl, int d, int Dr, int cl, int cr) {
  Carver c(nullptr);
  heff_ws(c, nm, Dl, d, Dr, cl, cr);
  return c.off;
}

static RnsView view_r(const double2* r, int Dr, int chi) { return {r, 1, (long)chi * Dr, 0}; }
static RnsView view_l(const double2* l, int Dl) { return {l, 1, Dl, 0}; }

ptn_status heff_prepare_rns(int nm, const double2* l, const double2* r, int Dl, int d, int Dr,
                            int cl, int cr, void* ws, size_t ws_bytes, cudaStream_t st) {
  auto layout = [&](Carver& c) { return heff_ws(c, nm, Dl, d, Dr, cl, cr); };
  RNS_CHECK_WS(layout);
  Carver c(ws);
  const HeffWs h = layout(c);
  PTN_TRY(rns_convert(view_r(r, Dr, cr), h.r, false, nullptr, st));
  return rns_convert(view_l(l, Dl), h.l, false, nullptr, st);
}

ptn_status heff_apply_rns(int nm, const double2* x, double2* y, const double2* w, const double2* l,
                          const double2* r, int Dl, int d, int Dr, int cl, int cr, void* ws,
                          const int* skip, cudaStream_t st) {
  Carver c(ws);
  const HeffWs h = heff_ws(c, nm, Dl, d, Dr, cl, cr);
  const RnsView vx{x, Dr, 1, 0}, vt{h.T2, 1, (long)d * Dr, 0};
  PTN_TRY(rns_convert(vx, h.x, false, skip, st, h.t2.e, h.t2.rows));
  // T2[l0,(wl,s),r2] = sum_(t,wr) W[(wl,s),(t,wr)] T1[l0,(t,wr),r2]
  const RnsStage s{w, (long)d * cr, 1, Dl, d * cr, cr, cl * d, Dr, h.T2, h.t2.e, d, false};
  PTN_TRY(rns_gemm_stage(h.x, vx, h.r, view_r(r, Dr, cr), s, h.res, skip, st));
  PTN_TRY(rns_convert(vt, h.t2, true, skip, st));
  return rns_gemm(h.l, view_l(l, Dl), h.t2, vt, ONE, ZERO, y, (long)d * Dr, h.res, skip, st);
}

// ================================================================ bond operator
size_t bond_workspace_bytes_rns(int nm, int Dl, int Dr, int chi) {
  Carver c(nullptr);
  bond_ws(c, nm, Dl, Dr, chi);
  return c.off;
}

ptn_status bond_prepare_rns(int nm, const double2* l, const double2* r, int Dl, int Dr, int chi,
                            void* ws, size_t ws_bytes, cudaStream_t st) {
  auto layout = [&](Carver& c) { return bond_ws(c, nm, Dl, Dr, chi); };
  RNS_CHECK_WS(layout);
  Carver c(ws);
  const BondWs b = layout(c);
  PTN_TRY(rns_convert(view_r(r, Dr, chi), b.r, false, nullptr, st));
  return rns_convert(view_l(l, Dl), b.l, false, nullptr, st);
}

ptn_status bond_apply_rns(int nm, const double2* x, double2* y, const double2* l, const double2* r,
                          int Dl, int Dr, int chi, void* ws, const int* skip, cudaStream_t st) {
  Carver c(ws);
  const BondWs b = bond_ws(c, nm, Dl, Dr, chi);
  const RnsView vx{x, Dr, 1, 0}, vt{b.T1, 1, Dr, 0};
  PTN_TRY(rns_convert(vx, b.x, false, skip, st));
  // T1[l0][(w, r2)]
  PTN_TRY(rns_gemm(b.x, vx, b.r, view_r(r, Dr, chi), ONE, ZERO, b.T1, (long)chi * Dr, b.res, skip,
                   st));
  // rows r2, terms (l0, w)
  PTN_TRY(rns_convert(vt, b.t1, false, skip, st));
  return rns_gemm(b.l, view_l(l, Dl), b.t1, vt, ONE, ZERO, y, Dr, b.res, skip, st);
}

// ================================================================ environments
size_t env_workspace_bytes_rns(int nm, int Dl, int d, int Dr, int cl, int cr) {
  Carver a(nullptr), b(nullptr);
  env_left_ws(a, nm, Dl, d, Dr, cl, cr);
  env_right_ws(b, nm, Dl, d, Dr, cl, cr);
  return std::max(a.off, b.off);
}

// l_next[ra, wr, rb] = sum A[l0,s,ra] W[wl,t,s,wr] L[l0,wl,l2] conj(B[l2,t,rb])
ptn_status env_left_rns(int nm, const double2* a, const double2* b, const double2* w,
                        const double2* l, double2* lnext, int Dl, int d, int Dr, int cl, int cr,
                        void* ws, size_t ws_bytes, cudaStream_t st) {
  auto layout = [&](Carver& c) { return env_left_ws(c, nm, Dl, d, Dr, cl, cr); };
  RNS_CHECK_WS(layout);
  Carver c(ws);
  const EnvWs e = layout(c);
  const RnsView v1{l, Dl, 1, 0}, v2{b, 1, (long)d * Dr, 1}, v3{a, 1, Dr, 0},
      v4{e.T2, 1, (long)cr * Dr, 0};
  PTN_TRY(rns_convert(v1, e.a1, false, nullptr, st, e.b2.e, e.b2.rows));
  PTN_TRY(rns_convert(v2, e.b1, false, nullptr, st));
  PTN_TRY(rns_convert(v3, e.a2, false, nullptr, st));
  // T2[l0,(s,wr),rb] = sum_(wl,t) W[wl,t,s,wr] T1[l0,(wl,t),rb]   (stage matrix W^T)
  const RnsStage s{w, 1, (long)d * cr, Dl, cl * d, d, d * cr, Dr, e.T2, e.b2.e, cr, false};
  PTN_TRY(rns_gemm_stage(e.a1, v1, e.b1, v2, s, e.res, nullptr, st));
  PTN_TRY(rns_convert(v4, e.b2, true, nullptr, st));
  return rns_gemm(e.a2, v3, e.b2, v4, ONE, ZERO, lnext, (long)cr * Dr, e.res, nullptr, st);
}

// r_next[la, wl, lb] = sum A[la,s,r0] W[wl,t,s,wr] R[r0,wr,r2] conj(B[lb,t,r2])
ptn_status env_right_rns(int nm, const double2* a, const double2* b, const double2* w,
                         const double2* r, double2* rnext, int Dl, int d, int Dr, int cl, int cr,
                         void* ws, size_t ws_bytes, cudaStream_t st) {
  auto layout = [&](Carver& c) { return env_right_ws(c, nm, Dl, d, Dr, cl, cr); };
  RNS_CHECK_WS(layout);
  Carver c(ws);
  const EnvWs e = layout(c);
  const RnsView v1{a, Dr, 1, 0}, v2 = view_r(r, Dr, cr), v3{e.T2, (long)d * Dr, 1, 0},
      v4{b, (long)d * Dr, 1, 1};
  PTN_TRY(rns_convert(v1, e.a1, false, nullptr, st, e.a2.e, e.a2.rows));
  PTN_TRY(rns_convert(v2, e.b1, false, nullptr, st));
  PTN_TRY(rns_convert(v4, e.b2, false, nullptr, st));
  // T2[l0,(wl,t),r2] = sum_(s,wr) W[(wl,t),(s,wr)] T1[l0,(s,wr),r2]
  const RnsStage s{w, (long)d * cr, 1, Dl, d * cr, cr, cl * d, Dr, e.T2, e.a2.e, d, true};
  PTN_TRY(rns_gemm_stage(e.a1, v1, e.b1, v2, s, e.res, nullptr, st));
  PTN_TRY(rns_convert(v3, e.a2, true, nullptr, st));
  return rns_gemm(e.a2, v3, e.b2, v4, ONE, ZERO, rnext, Dl, e.res, nullptr, st);
}

// ================================================================ plain GEMM
size_t zgemm_rns_workspace_bytes(int nm, long M, long N, long K) {
  Carver c(nullptr);
  c.operand(M, K, nm);
  c.operand(N, K, nm);
  c.take(rns_out_bytes(M, N, nm));
  return c.off + 256;
}

ptn_status zgemm_rns(int nm, const GemmArgs& g, void* ws, cudaStream_t st) {
  Carver c(reinterpret_cast<void*>(al(reinterpret_cast<uintptr_t>(ws))));
  const RnsOperand A = c.operand(g.M, g.K, nm);
  const RnsOperand B = c.operand(g.N, g.K, nm);
  void* res = c.take(0);
  // op(A) by rows, op(B) by columns
  const bool ta = g.opA == 'T' || g.opA == 'H', tb = g.opB == 'T' || g.opB == 'H';
  const bool ca = g.opA == 'C' || g.opA == 'H', cb = g.opB == 'C' || g.opB == 'H';
  const RnsView va = ta ? RnsView{g.A, 1, g.lda, ca} : RnsView{g.A, g.lda, 1, ca};
  const RnsView vb = tb ? RnsView{g.B, g.ldb, 1, cb} : RnsView{g.B, 1, g.ldb, cb};
  PTN_TRY(rns_convert(va, A, false, g.skip, st));
  PTN_TRY(rns_convert(vb, B, false, g.skip, st));
  return rns_gemm(A, va, B, vb, g.alpha, g.beta, g.C, g.ldc, res, g.skip, st);
}

}  // namespace ptn
