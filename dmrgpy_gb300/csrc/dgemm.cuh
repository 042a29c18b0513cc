// FP64 matrix products on the tensor cores by exact digit products (dgemm.cu).
#pragma once
#include "common.cuh"

namespace dmrg {

// One operand of C[M][N] = sum_k A[m][k] B[n][k]: element (row, k) of the
// FP64 / complex FP64 array p at row and k strides (outer, inner), in
// elements.  rows and K count elements (complex: complex elements).
struct DgOperand {
  const void* p;
  Ax2 rows, K;
  St2 sr, sk;
  int conj;
};

// Where a product's bounded waits record that one gave up, in device memory
// of the caller's: cleared by the split it is given to, or by the caller.  A
// product whose waits gave up leaves nan in its output.
struct DgStatus {
  int err;
  unsigned mark;   // DG_CLEARED once a split has cleared it
};
constexpr unsigned DG_CLEARED = 0x64675f30u;
constexpr size_t DG_STATUS_BYTES = 1024;
// DMRG_ERR_TIMEOUT if a product recorded one since (synchronises); with
// `marked` only where the word has been cleared by a split
int dg_gave_up(const DgStatus* st, bool marked, cudaStream_t s);

// Digit form of an operand in device memory: row exponents, then the digit
// blocks.  side 0: the M side (tiles of 128 rows), side 1: the N side (64).
size_t dg_bytes(int side, bool cplx_, long long rows, long long K);
template <typename T> int dg_split(int side, const DgOperand& o, void* buf, DgStatus* clear, cudaStream_t s);
// both operands in one launch: A on side 0, B on side 1
template <typename T>
int dg_split2(const DgOperand& A, void* bufa, const DgOperand& B, void* bufb, DgStatus* clear, cudaStream_t s);

// C = alpha A B (+ C): alpha +1 or -1; C at (row, column) strides in elements.
struct DgOut {
  void* C;
  Ax2 M, N;
  St2 cm, cn;
  double alpha;
  int accumulate;
};
// (the operands themselves are read only for rows and columns with infinities)
template <typename T>
int dg_gemm(const DgOperand& A, const void* Adig, const DgOperand& B, const void* Bdig, const DgOut& out,
            DgStatus* st, cudaStream_t s);
// whether the digit product of this shape is faster than the FP64 pipe
// (one_split: the other operand's digits are kept from an earlier call)
bool dg_pays(bool cplx_, long long M, long long N, long long K, bool one_split);

// C = alpha A B (+ C) for one unbatched strided contraction: both operands
// split into work (dg_product_bytes), then multiplied.  st: the caller's, or
// null for one in work.
size_t dg_product_bytes(bool cplx_, long long M, long long N, long long K);
template <typename T> size_t dg_product_bytes(const TGemm& g);
template <typename T>
int dg_product(const TGemm& g, const T* A, const T* B, double alpha, int accumulate, T* C, void* work,
               DgStatus* st, cudaStream_t s);

// C = alpha A B (+ C), alpha 1 or -1: a digit product where that is faster
// and ws holds its operands, else on the FP64 pipe
int fgemm(const TGemm& g, double alpha, const double* A, const double* B, int accumulate, double* C, void* ws,
          size_t ws_bytes, DgStatus* st, cudaStream_t s);

}  // namespace dmrg
