// Complex GEMM in a residue number system on the tensor cores (kernels: rns.cu): the
// operand type and the launches the contractions are built from.
#pragma once

#include "ptn_common.cuh"
#include <cuda_bf16.h>

namespace ptn {

// Moduli of the FP64 form (53 bits and more, else the DMMA kernels: 8192 terms) and of the mixed
// form: its operators (40 bits and more up to 16384 terms, 39 beyond) and its environment steps
// (49 and more up to 8192 terms, 48 beyond). Environments stay Hermitian to FP64 level: with 40
// bits the chain ends, whose small Krylov spaces are exhausted, see residuals around the
// breakdown threshold 100 n eps (2e-13 against 9e-14 at bond 2), and whether a run stops there
// would depend on rounding.
constexpr int RNS_FP64 = 14;
constexpr int RNS_MIXED = 11;
constexpr int RNS_MIXED_ENV = 13;

// element (r, k) of a complex operand: src[r * sr + k * sk], conjugated if `conj`
struct RnsView {
  const double2* src;
  long sr, sk;
  int conj;
};

// a complex operand with `rows` rows and kc columns as 2 * nm residue planes
// [plane][rows][Kp] (BF16, Kp a multiple of 8), and the exponent of the largest component of
// every row (as rns.cu keeps it; 0: no non-zero entry)
struct RnsOperand {
  __nv_bfloat16* p;
  int* e;
  int rows, kc, nm;
  long Kp;
  long plane() const { return (long)rows * Kp; }
};

// Powers of two on the terms of a product (FP64 form): A[m, k] 2^t[k] and B[n, k] 2^-t[k] have
// the same product. Rows are fixed-point numbers, so operands that grow and decay against each
// other along k (the two sides of a bond in a gauge A D, D^-1 B) would lose the bits of the
// entries that count: relative error (Frobenius norm, scalings taken out) of A D times
// D^-1 R D^-1 at bond 64, |D| spread over 1e6 / 1e12: 1.0e-11 / 7.2e-6 without, 3e-16 with
// it (DMMA 3e-16). Where the sizes of both operands are known beforehand (o: of the other
// one), t is what keeps the error at 2^-bits per term of the largest |A[m, k] B[n, k]|, and 0
// where nothing is lost. An operator's planes are made before its vectors: t then comes
// from the operator alone, which it brings to one size along k, so that the error of (m, n) is
// 2^-bits per term of the largest |A[m, k] B[n', k]| over k and n', and further down by what
// B's row n lies below the others. Either way scalings of the terms, of the rows of A and of those
// of B cancel. Terms k = (o, i) of a bond o and an MPO bond i < in take t = f[o] + g[i]: in a
// channel as sparse as the identity a term of its own size says nothing about its bond.
// The exponents are a launch of their own: H_eff at bonds 250 x 256 110 -> 117 us, an
// environment step at 187 x 300 85 -> 90, at bonds of 1024 1 %.
// be, f, o: exponents of the terms of the operand that t comes from and of the other one (term k
// at o[(k / odiv) % omod]; null: not known). Null t: no scaling.
constexpr int RNS_INNER_MAX = 64;
constexpr int RNS_TERM_JOBS = 4;
struct RnsTerms {
  int *be, *f, *o, *t;
  int in, odiv, omod;
};

// an operand whose terms' exponents are wanted (in > 1: be relative to f)
struct RnsTermsOf {
  RnsView v;
  int rows, kc, in;
  int *be, *f;
};

// of up to RNS_TERM_JOBS operands, one launch
ptn_status rns_term_exps(const RnsTermsOf* of, int n, const int* skip, cudaStream_t st);

// bytes of the planes / exponents / GEMM residues, each to be 256-byte aligned
size_t rns_plane_bytes(long rows, long kc, int nm);
size_t rns_out_bytes(long M, long N, int nm);
RnsOperand rns_operand(void* planes, void* exps, long rows, long kc, int nm);

// bits that a row-scaled value keeps in products of K complex terms, or 0 when K is too
// long for the precision of the form
int rns_bits(long K, int nm);

// whether the FP64 form of C (M x N) = A B (K terms) takes the residue planes
bool rns_wanted(long M, long N, long K);

// view -> residue planes for products over all kc terms. `have_exp`: the row exponents are
// in d.e already (from rns_gemm_stage). Also zeroes clear[0 .. nclear). `source`: the operand
// that terms->be was taken from, which also forms terms->t (before the other one reads it).
ptn_status rns_convert(const RnsView& v, const RnsOperand& d, bool have_exp, const int* skip,
                       cudaStream_t st, int* clear = nullptr, int nclear = 0,
                       const RnsTerms* terms = nullptr, bool source = false);

// out[m * ldc + n] = alpha sum_k A[m, k] B[n, k] + beta out[m * ldc + n]; va / vb are the
// views the operands came from (rows with infinities or NaNs and results outside the normal
// FP64 range are multiplied from them directly), res the residue buffer
ptn_status rns_gemm(const RnsOperand& A, const RnsView& va, const RnsOperand& B, const RnsView& vb,
                    double2 alpha, double2 beta, double2* out, long ldc, void* res,
                    const int* skip, cudaStream_t st);

// MPO stage on a product: out[x, q, y] = sum_p W[q, p] in[x, p, y] (W at w[q * ldq + p * ldp]),
// in[x, p, y] = element ((x, p / pin), (p % pin, y)) of the product. e2 (zeroed before) takes
// the row exponents of the output as an operand with rows (q % eq, y), or (x, q / eq) if by_x,
// under the scaling t2 of its terms (x, q / eq), or (q % eq, y) (null: none).
struct RnsStage {
  const double2* w;
  long ldq, ldp;
  int X, P, pin, Q, Y;
  double2* out;
  int* e2;
  const int* t2;
  int eq;
  bool by_x;
};
ptn_status rns_gemm_stage(const RnsOperand& A, const RnsView& va, const RnsOperand& B,
                          const RnsView& vb, const RnsStage& s, void* res, const int* skip,
                          cudaStream_t st);

// Contractions through residue planes (rns_ops.cu), nm one of the counts above. The views
// of an operator's l and r stay in use between prepare and the applies.
size_t heff_workspace_bytes_rns(int nm, int Dl, int d, int Dr, int cl, int cr);
ptn_status heff_prepare_rns(int nm, const double2* l, const double2* r, int Dl, int d, int Dr,
                            int cl, int cr, void* ws, size_t ws_bytes, cudaStream_t st);
ptn_status heff_apply_rns(int nm, const double2* x, double2* y, const double2* w, const double2* l,
                          const double2* r, int Dl, int d, int Dr, int cl, int cr, void* ws,
                          const int* skip, cudaStream_t st);
size_t bond_workspace_bytes_rns(int nm, int Dl, int Dr, int chi);
ptn_status bond_prepare_rns(int nm, const double2* l, const double2* r, int Dl, int Dr, int chi,
                            void* ws, size_t ws_bytes, cudaStream_t st);
ptn_status bond_apply_rns(int nm, const double2* x, double2* y, const double2* l, const double2* r,
                          int Dl, int Dr, int chi, void* ws, const int* skip, cudaStream_t st);
size_t env_workspace_bytes_rns(int nm, int Dl, int d, int Dr, int cl, int cr);
ptn_status env_left_rns(int nm, const double2* a, const double2* b, const double2* w,
                        const double2* l, double2* lnext, int Dl, int d, int Dr, int cl, int cr,
                        void* ws, size_t ws_bytes, cudaStream_t st);
ptn_status env_right_rns(int nm, const double2* a, const double2* b, const double2* w,
                         const double2* r, double2* rnext, int Dl, int d, int Dr, int cl, int cr,
                         void* ws, size_t ws_bytes, cudaStream_t st);

// moduli of a contraction's residue planes at precision `prec`, 0: the DMMA kernels (contract.cu)
int heff_form(int prec, int Dl, int d, int Dr, int cl, int cr);
int bond_form(int prec, int Dl, int Dr, int chi);

// C = alpha op(A) op(B) + beta C through residue planes (alignment of ws: any)
size_t zgemm_rns_workspace_bytes(int nm, long M, long N, long K);
ptn_status zgemm_rns(int nm, const GemmArgs& g, void* ws, cudaStream_t st);

}  // namespace ptn
