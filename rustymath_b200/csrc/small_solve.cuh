// The plain solve of a small system in two launches (getrf.cu), for api.cu.
#pragma once
#include <cstdint>

#include <cuda_runtime.h>

namespace rm {

struct SmallSolveResults {
  unsigned status;  // the device status word
  int32_t flag;     // LuWork::regular
};
constexpr int kSmallSolveParts = 8;  // doubles at amax

bool small_plain_solve_f64(const double* a, double* w, int64_t ldw, int64_t n, const double* b, int64_t k, double* x,
                           int64_t* ipiv, int64_t* perm, double* amax, unsigned* status, SmallSolveResults* results,
                           cudaStream_t stream, int* st);

}  // namespace rm
