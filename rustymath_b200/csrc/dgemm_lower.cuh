// The symmetric rank-k update's product (dgemm.cu), for the Cholesky factorization.
#pragma once
#include <cstdint>

#include <cuda_runtime.h>

namespace rm {

// C = alpha A B^T + beta C on the tiles of the n x n C that reach its lower triangle (A and B n x k);
// the tiles strictly above it are not touched.
int dgemm_lower_device(int64_t n, int64_t k, double alpha, const double* a, int64_t lda, const double* b, int64_t ldb,
                       double beta, double* c, int64_t ldc, unsigned* status, cudaStream_t stream);

}  // namespace rm
