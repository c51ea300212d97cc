// C -= A B in FP64 accuracy on the tcgen05 tensor cores, real and complex:
// the trailing updates of the FP64 LU factorisations and of the transient
// system's inverse (digit_gemm.cu has the method and its error).
#pragma once

#include <stddef.h>

namespace peec {

// K of one update at most: every sum of digit products stays an integer
// below 2^24 (see digit_gemm.cu).
static const int kDigitMaxKReal = 256;
static const int kDigitMaxKCplx = 192;

// Scratch of the updates of one factorisation: the digits of A (m rows) and
// B (n columns) and the exponents of their rows, columns and inner scaling.
struct DigitScratch {
    void *a = nullptr, *b = nullptr;
    int *ea = nullptr, *eb = nullptr, *ef = nullptr;
    unsigned *exact = nullptr;  // entries of the last update done in FP64
    void *mask = nullptr;  // complex: the nonzero parts of rows and columns
    int m = 0, n = 0, k = 0;
    bool cplx = false;
    DigitScratch() = default;
    // false, with nothing allocated and no error recorded, where there is no memory
    // for it or it is beyond digit_scratch_limit()
    bool alloc(bool cplx_, int m_, int n_, int k_);
    void release();
    ~DigitScratch() { release(); }
    DigitScratch(const DigitScratch &) = delete;
    DigitScratch &operator=(const DigitScratch &) = delete;
};
size_t digit_scratch_bytes(bool cplx, size_t m, size_t n, size_t k);
// Bytes that a DigitScratch of the calling thread may take (no limit at first).
size_t &digit_scratch_limit();

// C (m x n, row-major, leading dimension ldc) -= A (m x k, lda) B (k x n,
// ldb); complex entries are interleaved {re, im} and the leading dimensions
// count entries.  C must not overlap A or B.  m, n, k within the scratch's
// sizes.  *code (device): nothing is done when it is not 0; it is set to 6
// when a bounded wait inside the kernel runs out, and to 7 when more than exact_limit
// entries were so small beside their rows and columns that FP64 FMAs did them
// (complex only; the update is complete all the same).
bool digit_gemm_sub(bool cplx, const void *A, size_t lda, const void *B, size_t ldb, void *C, size_t ldc, int m, int n,
                    int k, DigitScratch &s, int *code, size_t exact_limit = ~(size_t)0);

}  // namespace peec
