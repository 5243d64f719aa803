// Host build of the integer-pipe logarithm over its whole range
// (pihm-cuda_gb300/csrc/int_math.cuh) for the CPU tests.
#include <cstdint>

#include "int_math.cuh"

extern "C" void im_log_any(const double *x, double *out, int32_t *ok, int64_t n, int32_t ten) {
  for (int64_t i = 0; i < n; i++) ok[i] = pihm::im::log_any_i(x[i], ten != 0, out[i]) ? 1 : 0;
}
