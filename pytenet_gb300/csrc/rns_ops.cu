// Site / bond operators and environment steps (pytenet/chain_ops.py:16-99, 237-317) with both
// GEMMs of every contraction in the residue number system (rns.cu): the FP64 form where the
// problem is large enough for it (contract.cu decides), the mixed form nearly always.
//
// Data flow of H_eff . x (site tensors (Dl, d, Dr), MPO bonds cl / cr); an operand is a set
// of residue planes, rows x terms:
//   prepare (once per local step):  R -> rows (wr, r2), terms r0;  L -> rows l2, terms (l0, wl);
//           in the FP64 form the scaling of both GEMMs' terms comes from them (RnsTerms)
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
  // scaling of outer * inner terms from one operand
  RnsTerms terms(long outer, int inner, int nm) {
    RnsTerms t{nullptr, nullptr, nullptr, nullptr, 1, 1, 1};
    if (nm != RNS_FP64) return t;
    if (inner <= RNS_INNER_MAX) t.in = inner;
    t.be = static_cast<int*>(take((size_t)outer * inner * sizeof(int)));
    t.f = static_cast<int*>(take((size_t)outer * sizeof(int)));
    t.t = static_cast<int*>(take((size_t)outer * inner * sizeof(int)));
    return t;
  }
  // from both, the other one's term k at (k / odiv) % omod
  RnsTerms terms_of_both(long kc, int odiv, int omod, int nm) {
    RnsTerms t = terms(kc, 1, nm);
    if (nm != RNS_FP64) return t;
    t.o = static_cast<int*>(take((size_t)omod * sizeof(int)));
    t.odiv = odiv;
    t.omod = omod;
    return t;
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
  RnsTerms tr, tl;        // from R and L
  double2* T2;
  void* res;
};

HeffWs heff_ws(Carver& c, int nm, int Dl, int d, int Dr, int cl, int cr) {
  HeffWs w;
  w.r = c.operand((long)cr * Dr, Dr, nm);
  w.l = c.operand(Dl, (long)Dl * cl, nm);
  w.x = c.operand((long)Dl * d, Dr, nm);
  w.t2 = c.operand((long)d * Dr, (long)Dl * cl, nm);
  w.tr = c.terms(Dr, 1, nm);
  w.tl = c.terms(Dl, cl, nm);
  w.T2 = static_cast<double2*>(c.take((size_t)Dl * cl * d * Dr * sizeof(double2)));
  w.res = c.take(std::max(rns_out_bytes((long)Dl * d, (long)cr * Dr, nm),
                          rns_out_bytes(Dl, (long)d * Dr, nm)));
  return w;
}

struct BondWs {
  RnsOperand r, l, x, t1;
  RnsTerms tr, tl;
  double2* T1;
  void* res;
};

BondWs bond_ws(Carver& c, int nm, int Dl, int Dr, int chi) {
  BondWs w;
  w.r = c.operand((long)chi * Dr, Dr, nm);
  w.l = c.operand(Dl, (long)Dl * chi, nm);
  w.x = c.operand(Dl, Dr, nm);
  w.t1 = c.operand(Dr, (long)Dl * chi, nm);
  w.tr = c.terms(Dr, 1, nm);
  w.tl = c.terms(Dl, chi, nm);
  w.T1 = static_cast<double2*>(c.take((size_t)Dl * chi * Dr * sizeof(double2)));
  w.res = c.take(std::max(rns_out_bytes(Dl, (long)chi * Dr, nm), rns_out_bytes(Dl, Dr, nm)));
  return w;
}

// a1 b1: first GEMM, a2 b2: second one
struct EnvWs {
  RnsOperand a1, b1, a2, b2;
  RnsTerms t1, t2;        // scaling of their terms; of T2 the sizes that L (R) gives its terms
  double2* T2;
  void* res;
};

EnvWs env_left_ws(Carver& c, int nm, int Dl, int d, int Dr, int cl, int cr) {
  EnvWs w;
  w.a1 = c.operand((long)Dl * cl, Dl, nm);             // L, rows (l0, wl), terms l2
  w.b1 = c.operand((long)d * Dr, Dl, nm);              // conj(B), rows (t, rb), terms l2
  w.a2 = c.operand(Dr, (long)Dl * d, nm);              // A, rows ra, terms (l0, s)
  w.b2 = c.operand((long)cr * Dr, (long)Dl * d, nm);   // T2, rows (wr, rb), terms (l0, s)
  w.t1 = c.terms_of_both(Dl, 1, Dl, nm);
  w.t2 = c.terms_of_both((long)Dl * d, d, Dl, nm);
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
  w.t1 = c.terms_of_both(Dr, 1, Dr, nm);
  w.t2 = c.terms_of_both((long)d * Dr, 1, Dr, nm);
  w.T2 = static_cast<double2*>(c.take((size_t)Dl * cl * d * Dr * sizeof(double2)));
  w.res = c.take(std::max(rns_out_bytes((long)Dl * d, (long)cr * Dr, nm),
                          rns_out_bytes((long)Dl * cl, Dl, nm)));
  return w;
}

RnsTermsOf source_terms(const RnsView& v, const RnsOperand& o, const RnsTerms& t) {
  return {v, o.rows, o.kc, t.in, t.be, t.f};
}

// the other operand's, `rows` of them to each of t.omod terms
RnsTermsOf other_terms(const RnsView& v, long rows, const RnsTerms& t) {
  return {v, (int)rows, t.omod, 1, t.o, nullptr};
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
  const RnsView vr = view_r(r, Dr, cr), vl = view_l(l, Dl);
  if (h.tr.t != nullptr) {
    const RnsTermsOf of[2] = {source_terms(vr, h.r, h.tr), source_terms(vl, h.l, h.tl)};
    PTN_TRY(rns_term_exps(of, 2, nullptr, st));
  }
  PTN_TRY(rns_convert(vr, h.r, false, nullptr, st, nullptr, 0, &h.tr, true));
  return rns_convert(vl, h.l, false, nullptr, st, nullptr, 0, &h.tl, true);
}

ptn_status heff_apply_rns(int nm, const double2* x, double2* y, const double2* w, const double2* l,
                          const double2* r, int Dl, int d, int Dr, int cl, int cr, void* ws,
                          const int* skip, cudaStream_t st) {
  Carver c(ws);
  const HeffWs h = heff_ws(c, nm, Dl, d, Dr, cl, cr);
  const RnsView vx{x, Dr, 1, 0}, vt{h.T2, 1, (long)d * Dr, 0};
  PTN_TRY(rns_convert(vx, h.x, false, skip, st, h.t2.e, h.t2.rows, &h.tr));
  // T2[l0,(wl,s),r2] = sum_(t,wr) W[(wl,s),(t,wr)] T1[l0,(t,wr),r2]
  const RnsStage s{w, (long)d * cr, 1, Dl, d * cr, cr, cl * d, Dr, h.T2, h.t2.e, h.tl.t, d,
                   false};
  PTN_TRY(rns_gemm_stage(h.x, vx, h.r, view_r(r, Dr, cr), s, h.res, skip, st));
  PTN_TRY(rns_convert(vt, h.t2, true, skip, st, nullptr, 0, &h.tl));
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
  const RnsView vr = view_r(r, Dr, chi), vl = view_l(l, Dl);
  if (b.tr.t != nullptr) {
    const RnsTermsOf of[2] = {source_terms(vr, b.r, b.tr), source_terms(vl, b.l, b.tl)};
    PTN_TRY(rns_term_exps(of, 2, nullptr, st));
  }
  PTN_TRY(rns_convert(vr, b.r, false, nullptr, st, nullptr, 0, &b.tr, true));
  return rns_convert(vl, b.l, false, nullptr, st, nullptr, 0, &b.tl, true);
}

ptn_status bond_apply_rns(int nm, const double2* x, double2* y, const double2* l, const double2* r,
                          int Dl, int Dr, int chi, void* ws, const int* skip, cudaStream_t st) {
  Carver c(ws);
  const BondWs b = bond_ws(c, nm, Dl, Dr, chi);
  const RnsView vx{x, Dr, 1, 0}, vt{b.T1, 1, Dr, 0};
  PTN_TRY(rns_convert(vx, b.x, false, skip, st, nullptr, 0, &b.tr));
  // T1[l0][(w, r2)]
  PTN_TRY(rns_gemm(b.x, vx, b.r, view_r(r, Dr, chi), ONE, ZERO, b.T1, (long)chi * Dr, b.res, skip,
                   st));
  // rows r2, terms (l0, w)
  PTN_TRY(rns_convert(vt, b.t1, false, skip, st, nullptr, 0, &b.tl));
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
  if (e.t1.t != nullptr) {
    // T2's terms (l0, s) are as large as L at l0
    const RnsTermsOf of[4] = {source_terms(v2, e.b1, e.t1), other_terms(v1, e.a1.rows, e.t1),
                              source_terms(v3, e.a2, e.t2),
                              other_terms({l, 1, (long)cl * Dl, 0}, (long)cl * Dl, e.t2)};
    PTN_TRY(rns_term_exps(of, 4, nullptr, st));
  }
  PTN_TRY(rns_convert(v2, e.b1, false, nullptr, st, e.b2.e, e.b2.rows, &e.t1, true));
  PTN_TRY(rns_convert(v1, e.a1, false, nullptr, st, nullptr, 0, &e.t1));
  PTN_TRY(rns_convert(v3, e.a2, false, nullptr, st, nullptr, 0, &e.t2, true));
  // T2[l0,(s,wr),rb] = sum_(wl,t) W[wl,t,s,wr] T1[l0,(wl,t),rb]   (stage matrix W^T)
  const RnsStage s{w, 1, (long)d * cr, Dl, cl * d, d, d * cr, Dr, e.T2, e.b2.e, e.t2.t, cr,
                   false};
  PTN_TRY(rns_gemm_stage(e.a1, v1, e.b1, v2, s, e.res, nullptr, st));
  PTN_TRY(rns_convert(v4, e.b2, true, nullptr, st, nullptr, 0, &e.t2));
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
  if (e.t1.t != nullptr) {
    // T2's terms (t, r2) are as large as R at r2
    const RnsTermsOf of[4] = {source_terms(v1, e.a1, e.t1), other_terms(v2, e.b1.rows, e.t1),
                              source_terms(v4, e.b2, e.t2),
                              other_terms({r, Dr, 1, 0}, (long)Dr * cr, e.t2)};
    PTN_TRY(rns_term_exps(of, 4, nullptr, st));
  }
  PTN_TRY(rns_convert(v1, e.a1, false, nullptr, st, e.a2.e, e.a2.rows, &e.t1, true));
  PTN_TRY(rns_convert(v2, e.b1, false, nullptr, st, nullptr, 0, &e.t1));
  PTN_TRY(rns_convert(v4, e.b2, false, nullptr, st, nullptr, 0, &e.t2, true));
  // T2[l0,(wl,t),r2] = sum_(s,wr) W[(wl,t),(s,wr)] T1[l0,(s,wr),r2]
  const RnsStage s{w, (long)d * cr, 1, Dl, d * cr, cr, cl * d, Dr, e.T2, e.a2.e, e.t2.t, d,
                   true};
  PTN_TRY(rns_gemm_stage(e.a1, v1, e.b1, v2, s, e.res, nullptr, st));
  PTN_TRY(rns_convert(v3, e.a2, true, nullptr, st, nullptr, 0, &e.t2));
  return rns_gemm(e.a2, v3, e.b2, v4, ONE, ZERO, rnext, Dl, e.res, nullptr, st);
}

// ================================================================ plain GEMM
size_t zgemm_rns_workspace_bytes(int nm, long M, long N, long K) {
  Carver c(nullptr);
  c.operand(M, K, nm);
  c.operand(N, K, nm);
  c.terms_of_both(K, 1, (int)K, nm);
  c.take(rns_out_bytes(M, N, nm));
  return c.off + 256;
}

ptn_status zgemm_rns(int nm, const GemmArgs& g, void* ws, cudaStream_t st) {
  Carver c(reinterpret_cast<void*>(al(reinterpret_cast<uintptr_t>(ws))));
  const RnsOperand A = c.operand(g.M, g.K, nm);
  const RnsOperand B = c.operand(g.N, g.K, nm);
  const RnsTerms terms = c.terms_of_both(g.K, 1, g.K, nm);
  void* res = c.take(0);
  // op(A) by rows, op(B) by columns
  const bool ta = g.opA == 'T' || g.opA == 'H', tb = g.opB == 'T' || g.opB == 'H';
  const bool ca = g.opA == 'C' || g.opA == 'H', cb = g.opB == 'C' || g.opB == 'H';
  const RnsView va = ta ? RnsView{g.A, 1, g.lda, ca} : RnsView{g.A, g.lda, 1, ca};
  const RnsView vb = tb ? RnsView{g.B, g.ldb, 1, cb} : RnsView{g.B, 1, g.ldb, cb};
  // which operand forms the scaling of the terms makes no difference: the shorter one
  const bool from_b = g.N <= g.M;
  if (terms.t != nullptr) {
    const RnsTermsOf of[2] = {source_terms(from_b ? vb : va, from_b ? B : A, terms),
                              other_terms(from_b ? va : vb, from_b ? g.M : g.N, terms)};
    PTN_TRY(rns_term_exps(of, 2, g.skip, st));
  }
  if (from_b) PTN_TRY(rns_convert(vb, B, false, g.skip, st, nullptr, 0, &terms, true));
  PTN_TRY(rns_convert(va, A, false, g.skip, st, nullptr, 0, &terms, !from_b));
  if (!from_b) PTN_TRY(rns_convert(vb, B, false, g.skip, st, nullptr, 0, &terms));
  return rns_gemm(A, va, B, vb, g.alpha, g.beta, g.C, g.ldc, res, g.skip, st);
}

}  // namespace ptn
