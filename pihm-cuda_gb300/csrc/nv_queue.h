// A queue of N_Vector operations over the vectors of one family, for the
// integrator (bdf.cpp).  It issues far more element-wise operations than it
// reads values back, so they are collected until a value is needed -- by a
// reduction, a right-hand side, the caller -- and then run in one kernel,
// entry by entry in the order they were issued, with the reduction that ended
// them (nvector.cu, k_seq).  Every entry, norm and slot is the one the
// separate kernels give, bit for bit.
//
// Whatever the queue does not take (a vector of another family or length, an
// operation the caller replaced in the vector's table) makes the call return
// false; the caller then flushes and calls the table.
//
// A launch that fails loses what was queued, so every value asked for from
// then on is NAN (a fetch fails) until the caller has taken the failure
// (take_failure), whichever launch it was.
#pragma once

#include <cstdint>

#include "nv_select.h"
#include "pihm_nvector.h"

namespace pihm_nv {

struct Family;

// Kernel parameters: the operations, then up to two reductions.
constexpr int kSeqOps = 24;
// Operand bits of SeqOp::fwd and SeqRed::fwd: the operand is the result of
// the operation before.  SEQ_DEAD: a later operation of the sequence
// overwrites the result before anything else reads it, so it is not stored.
enum : uint8_t { SEQ_X = 1, SEQ_Y = 2, SEQ_Z = 4, SEQ_DEAD = 8 };

struct SeqOp {
  const double *x, *y;
  double *z;
  double a, b;
  uint8_t code;  // EwOp, or EW_COUNT: a linear sum with coefficients from slots
  uint8_t fwd, ka, sa, kb, sb, ztag, pad;
};

struct SeqRed {
  const double *x, *y;
  double *out;       // value and flag
  int64_t wrms_n;    // > 0: the WRMS norm instead of the sum
  int32_t op;        // -1 none
  uint8_t fwd;
};

struct Seq {
  int64_t n;
  int32_t nops, nred;
  double *partials;
  const double *slots;
  unsigned int *ticket;
  double *host;                // with a sequence number: the reductions' values go
  uint64_t *host_seq;          // to host[0..1], and slots 0..fetch-1 and *word
  uint64_t seq;                // behind them
  const unsigned int *word;
  int32_t fetch;
  SeqRed red[2];
  SeqOp op[kSeqOps];
};

class NvQueue {
 public:
  bool linear_sum(double a, N_Vector x, double b, N_Vector y, N_Vector z);
  bool linear_sum_coef(const pihm_nv_coef &a, N_Vector x, const pihm_nv_coef &b, N_Vector y, N_Vector z);
  bool scale(double c, N_Vector x, N_Vector z);
  // op: EW_CONST (b unused), EW_ABS, EW_INV, EW_DIV, EW_PROD, EW_ADDCONST;
  // x and y may be null where the operation does not read them
  bool ew(int op, double a, double b, N_Vector x, N_Vector y, N_Vector z);
  // op: R_DOT, R_MAXABS, R_WSQ, R_MIN: queued, run, *value the reduction
  // (NAN when the device failed, as the vector's own operation gives)
  bool reduce(int op, N_Vector x, N_Vector y, double *value);
  // Whether the queue takes v at all.
  bool accepts(N_Vector v) const;
  // min(m) and the sum of squares of x * w after the queued work, or (m
  // null) the sum alone; dev_word (may be null): a device word read with them
  bool min_wsq(N_Vector m, N_Vector x, N_Vector w, double *mn, double *sum, const unsigned int *dev_word,
               unsigned int *word_out);
  // R_DOT, or R_WSQ as the WRMS norm, left in a slot
  bool reduce_slot(int op, N_Vector x, N_Vector y, int slot);
  // N_VFetchSlots_PihmGpu with the queued work ahead of it
  bool fetch(N_Vector v, int count, double *out, const unsigned int *dev_word, unsigned int *word_out, int *rc);
  int flush();
  // whether a launch has failed since the last call
  bool take_failure() {
    const bool f = failed;
    failed = false;
    return f;
  }
  bool empty() const { return q.nops == 0 && q.nred == 0; }

 private:
  bool take(N_Vector z, N_Vector x, N_Vector y);
  void push(const SeqOp &o);
  void push_red(const SeqRed &r);
  // Run what is queued.  back: the reductions' values come to the host with
  // the launch, and behind them `fetch` slots (-1 none) and *word (may be
  // null); whatever a launch hands back is its own, not the one before's.
  int launch(bool back, int fetch = -1, const unsigned int *word = nullptr);
  Family *fam = nullptr;
  bool failed = false;
  Seq q{};
};

}  // namespace pihm_nv
