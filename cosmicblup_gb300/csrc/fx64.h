// FP64-accurate dense algebra on the tensor cores by exact fixed-point digits
// (fx64.cu): products, Cholesky factors and SPD inverses of the set-up and
// dense-AI paths.
#pragma once
#include <cstdint>
#include <functional>
#include "devbuf.h"

struct cbx_handle;

namespace cbx {

// Digits of an operand: rows (padded to 128) x k (padded to 32), 16 bytes an entry.
struct FxPanel {
  DevBuf<uint8_t> dig;
  DevBuf<int32_t> ex;
  int rt = 0, ks = 0;  // row tiles of 128, K steps of 32
};

// Rows of P from src: element (r, k) is src[r * ld + k], or src[k * ld + r] when
// trans.
void fx64_digits(cbx_handle* h, FxPanel& P, const double* src, int64_t ld, int64_t rows, int64_t k, bool trans);
// the same for rows of src as they lie, or false where the digits do not fit the memory
bool fx64_try_digits(cbx_handle* h, FxPanel& P, const double* src, int64_t ld, int64_t rows, int64_t k);
// C[i * ldc + j] = sum_k A(i, k) B(j, k) for i < m, j < n.
void fx64_gemm(cbx_handle* h, const FxPanel& A, const FxPanel& B, int64_t m, int64_t n, double* C, int64_t ldc);

// C = A B' for n x n row-major matrices.  Ad and Bd take the digits (B's are there already when
// has_b); where they do not fit, the product goes by groups of rows, with the same bits.
// Returns whether Bd holds the digits of B.
bool fx64_matmul(cbx_handle* h, const double* A, FxPanel& Ad, const double* B, FxPanel& Bd, bool has_b, int64_t n,
                 double* C);

// out[i * os + c] = sum_k Q(i, k) X[(p + gmap[k]) * xs + c] for i < ng, c < ncols <= 64, zero
// for ncols <= c < oc.  Q holds the digits of the ng x ng block; V and part are scratch.
// Does nothing while active (may be null) points to 0.  before (may be empty) is called ahead
// of the MMAs: true if its last launch lets them start with it (release_successor).
void fx64_product(cbx_handle* h, const FxPanel& Q, FxPanel& V, DevBuf<double>& part, const double* X, int xs, int64_t p,
                  const int32_t* gmap, int64_t ng, int ncols, double* out, int os, int oc, const int* active,
                  const std::function<bool()>& before = {});

// diag I + all 11' is added to a matrix on reading it
struct FxAdd {
  double diag = 0.0, all = 0.0;
};

// Cholesky of the symmetric n x n matrix A (column-major, its lower triangle is
// read).  Needs 8 n^2 bytes beside A and out, and up to 8 n^2 more for an inverse where the
// memory has them.  Returns false when a pivot is not positive.  logdet (may be null) gets
// log det A.  With inverse, out (may be A) receives the full symmetric A^-1;
// otherwise, when out is given, out gets the factor U = L' (column-major upper
// triangle, zeros below).
bool fx64_cholesky(cbx_handle* h, const double* A, int64_t n, bool inverse, double* out, double* logdet,
                   FxAdd add = {});

// y[i] = (hi[i] 2^32 + lo[i]) 2^e[i], |e[i]| < 900 (self-test of the products' conversion)
void fx64_selftest_totals(cbx_handle* h, const int64_t* hi, const int64_t* lo, const int32_t* e, int64_t n, double* y);

}  // namespace cbx
