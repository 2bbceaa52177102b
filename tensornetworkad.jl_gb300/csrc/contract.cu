// Pairwise tensor contraction on the device: the role OMEinsum's ein"..." plays
// in the reference (e.g. src/ctmrg.jl:130-140, src/variationalipeps.jl:52).
// A contraction is mapped to one GEMM: free labels of A become the rows, free
// labels of B the columns, shared labels the inner dimension.  The DFMA GEMM
// reads and writes tensors in any label order.  For the tensor-core GEMMs and
// large matrix-vector products, operands whose memory order already matches a
// (transposed) matrix view are used in place and others packed by one permutation
// kernel, and the output is permuted when the requested label order interleaves
// A's and B's free labels.
#include <cstring>
#include <string>

#include "tnad_internal.h"

namespace tnad {

static int find_label(const char* s, char ch) {
  for (int i = 0; s[i]; ++i)
    if (s[i] == ch) return i;
  return -1;
}

Ten contract_shape(const Ten& A, const char* la, const Ten& B, const char* lb, const char* lc) {
  Ten C;
  C.nd = (int)strlen(lc);
  for (int k = 0; k < C.nd; ++k) {
    int ia = find_label(la, lc[k]);
    int ib = find_label(lb, lc[k]);
    TNAD_REQUIRE(ia >= 0 || ib >= 0, TNAD_ERR_ARG, std::string("contract: output label not in inputs: ") + lc);
    C.dim[k] = ia >= 0 ? A.dim[ia] : B.dim[ib];
  }
  return C;
}

// Is `have` (labels in memory order) equal to the concatenation x+y ?
static bool is_concat(const std::string& have, const std::string& x, const std::string& y) { return have == x + y; }

static void perm_to(tnad_ctx* c, const Ten& T, const std::string& have, const std::string& want, double* out) {
  int perm[10];
  for (size_t k = 0; k < want.size(); ++k) perm[k] = (int)have.find(want[k]);
  permute(c, T, perm, out);
}

// Extents and strides of the labels `sel` (first fastest) in a tensor stored with
// labels `have`; labels adjacent in memory merge.  false: more than kMax extents.
static bool label_map(const int64_t* dim, const std::string& have, const std::string& sel, GemmMap& m) {
  m.nd = 0;
  for (char ch : sel) {
    const size_t k = have.find(ch);
    int64_t stride = 1;
    for (size_t i = 0; i < k; ++i) stride *= dim[i];
    if (dim[k] == 1) continue;
    if (m.nd > 0 && m.str[m.nd - 1] * (int64_t)m.dim[m.nd - 1] == stride) {
      m.dim[m.nd - 1] *= (unsigned)dim[k];
      continue;
    }
    if (m.nd == GemmMap::kMax) return false;
    m.dim[m.nd] = (unsigned)dim[k];
    m.str[m.nd++] = stride;
  }
  if (m.nd == 0) {
    m.nd = 1;
    m.dim[0] = 1;
    m.str[0] = 1;
  }
  return true;
}

void contract(tnad_ctx* c, int prec, const Ten& A0, const char* la0, const Ten& B0, const char* lb0, Ten& C,
              const char* lc0, double alpha, double beta) {
  TNAD_REQUIRE((int)strlen(la0) == A0.nd && (int)strlen(lb0) == B0.nd, TNAD_ERR_ARG,
               std::string("contract: label/rank mismatch ") + la0 + "," + lb0);
  std::string la = la0, lb = lb0, lc = lc0;
  // shape check of shared labels
  for (size_t i = 0; i < la.size(); ++i) {
    int j = find_label(lb0, la[i]);
    if (j >= 0)
      TNAD_REQUIRE(A0.dim[i] == B0.dim[j], TNAD_ERR_SHAPE,
                   std::string("contract: dimension mismatch on label ") + la[i] + " in " + la0 + "," + lb0);
  }
  Ten shp = contract_shape(A0, la0, B0, lb0, lc0);
  C.nd = shp.nd;
  for (int k = 0; k < C.nd; ++k) C.dim[k] = shp.dim[k];
  for (char ch : la)
    TNAD_REQUIRE(lb.find(ch) != std::string::npos || lc.find(ch) != std::string::npos, TNAD_ERR_ARG,
                 "contract: summed-out label only in A (use a reduction)");
  for (char ch : lb)
    TNAD_REQUIRE(la.find(ch) != std::string::npos || lc.find(ch) != std::string::npos, TNAD_ERR_ARG,
                 "contract: summed-out label only in B (use a reduction)");
  for (char ch : lc)
    TNAD_REQUIRE(!(la.find(ch) != std::string::npos && lb.find(ch) != std::string::npos), TNAD_ERR_ARG,
                 "contract: batch labels are not supported");

  // Put the operand owning the first output label first.
  const Ten* A = &A0;
  const Ten* B = &B0;
  if (!lc.empty() && la.find(lc[0]) == std::string::npos) {
    std::swap(A, B);
    std::swap(la, lb);
  }
  std::string Ml, Nl, Kl;
  for (char ch : lc) (la.find(ch) != std::string::npos ? Ml : Nl) += ch;
  const Ten* big = A->numel() >= B->numel() ? A : B;
  const std::string& lbig = (big == A) ? la : lb;
  for (char ch : lbig)
    if (la.find(ch) != std::string::npos && lb.find(ch) != std::string::npos) Kl += ch;

  auto dims_of = [&](const Ten* T, const std::string& lab, const std::string& sel) {
    int64_t p = 1;
    for (char ch : sel) p *= T->dim[lab.find(ch)];
    return p;
  };
  int64_t M = dims_of(A, la, Ml), N = dims_of(B, lb, Nl), K = dims_of(A, la, Kl);

  // A matrix in memory times a vector: the GEMM's matrix-vector kernels read it once,
  // where a tile does 16 columns' multiply-adds for one.  They are the faster ones with
  // a thread per row from four 16-row tiles an SM on (20000×50: 99 µs against 122 by
  // tiles; 2000×2000: 686 against 322, a thread walks all of K), and by columns for up to
  // 32 of them and long K (20×10^5: 198 against 286; 32×8192: 100 against 95).
  const bool by_rows = is_concat(la, Ml, Kl), by_cols = is_concat(la, Kl, Ml);
  const bool gemv = N == 1 && (by_rows ? M >= 64 * (int64_t)c->sm_count : by_cols && M <= 32 && K >= 16384);
  if (M > 0 && N > 0 && K > 0 && !gemv && gemm_is_f64(c, prec, M, N, K)) {
    // DFMA tiles read and write the tensors in place, in any label order
    GemmMap am, ak, bk, bn, cm, cn;
    if (label_map(A->dim, la, Ml, am) && label_map(A->dim, la, Kl, ak) && label_map(B->dim, lb, Kl, bk) &&
        label_map(B->dim, lb, Nl, bn) && label_map(C.dim, lc, Ml, cm) && label_map(C.dim, lc, Nl, cn)) {
      gemm_f64_map(c, M, N, K, alpha, A->p, am, ak, B->p, bk, bn, beta, C.p, cm, cn);
      return;
    }
  }
  WsScope scope(c);
  const double* Ap = A->p;
  char ta = 'N';
  int64_t lda = M > 0 ? M : 1;
  if (by_rows) {
    ta = 'N';
    lda = M;
  } else if (by_cols) {
    ta = 'T';
    lda = K;
  } else {
    double* t = ws_d(c, A->numel());
    perm_to(c, *A, la, Ml + Kl, t);
    Ap = t;
  }
  const double* Bp = B->p;
  char tb = 'N';
  int64_t ldb = K;
  if (is_concat(lb, Kl, Nl)) {
    tb = 'N';
    ldb = K;
  } else if (is_concat(lb, Nl, Kl)) {
    tb = 'T';
    ldb = N;
  } else {
    double* t = ws_d(c, B->numel());
    perm_to(c, *B, lb, Kl + Nl, t);
    Bp = t;
  }
  if (lda < 1) lda = 1;
  if (ldb < 1) ldb = 1;
  if (lc == Ml + Nl) {
    gemm(c, prec, ta, tb, M, N, K, alpha, Ap, lda, Bp, ldb, beta, C.p, M > 0 ? M : 1);
  } else {
    double* t = ws_d(c, M * N);
    gemm(c, prec, ta, tb, M, N, K, 1.0, Ap, lda, Bp, ldb, 0.0, t, M > 0 ? M : 1);
    Ten T;
    T.p = t;
    std::string have = Ml + Nl;
    T.nd = (int)have.size();
    for (int k = 0; k < T.nd; ++k) {
      char ch = have[k];
      size_t ia = la.find(ch);
      T.dim[k] = ia != std::string::npos ? A->dim[ia] : B->dim[lb.find(ch)];
    }
    int perm[10];
    for (size_t k = 0; k < lc.size(); ++k) perm[k] = (int)have.find(lc[k]);
    permute(c, T, perm, C.p, alpha, beta);
  }
}

}  // namespace tnad
