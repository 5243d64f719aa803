// Host build of the integer-pipe exponential and logarithms
// (pihm-cuda_gb300/csrc/int_math.cuh) for the CPU tests.
#include <cstdint>

#include "int_math.cuh"

extern "C" {
// out[i] = e^x[i]; ok[i] = 0 where the integer path declines
void im_exp(const double *x, double *out, int32_t *ok, int64_t n) {
  for (int64_t i = 0; i < n; i++) ok[i] = pihm::im::exp_i(x[i], out[i]) ? 1 : 0;
}
// out[i] = ln x[i] (ten == 0) or log10 x[i]
void im_log(const double *x, double *out, int32_t *ok, int64_t n, int32_t ten) {
  const uint64_t c = ten ? kImCLog10 : kImCLn2;
  for (int64_t i = 0; i < n; i++) ok[i] = pihm::im::log_i(x[i], c, out[i]) ? 1 : 0;
}
// the same for x next to one
void im_log_near1(const double *x, double *out, int32_t *ok, int64_t n, int32_t ten) {
  for (int64_t i = 0; i < n; i++) ok[i] = pihm::im::log_near1_i(x[i], ten != 0, out[i]) ? 1 : 0;
}
// cos x for 0 <= x < 3.15
void im_cos(const double *x, double *out, int32_t *ok, int64_t n) {
  for (int64_t i = 0; i < n; i++) ok[i] = pihm::im::cos_i(x[i], out[i]) ? 1 : 0;
}
}
