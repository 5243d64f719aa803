// Derived from SUNDIALS 2.7.0 (CVODE 2.9.0). Copyright (c) 2002-2016,
// Lawrence Livermore National Security; produced at the Lawrence Livermore
// National Laboratory (UCRL-CODE-155951). Redistributed under the SUNDIALS
// BSD-3 licence: its full text, conditions and disclaimer are in
// pihm-cuda_gb300/NOTICE.SUNDIALS.
//
// Device-resident N_Vector (SUNDIALS 2.7 / CVODE 2.9 operations table) for
// sm_103a.  See include/pihm_nvector.h for the contract.
//
// Element-wise kernels use __dmul_rn/__dadd_rn so the compiler cannot fuse a
// multiply and an add: every element equals what the serial N_Vector computes
// (cvode/src/nvec_ser/nvector_serial.c:421-1060), including its special cases
// (a == 1, b == -1, a == b, ...) which change the rounding.
//
// Reductions: each block reduces a fixed, grid-strided slice of the vector
// with a warp-shuffle tree, writes one partial, and the last block to finish
// (atomic ticket) combines the partials in index order.  The grid size depends
// only on the length, so the result is identical from run to run.
#include <cfloat>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>

#include "host_flag.h"
#include "nv_queue.h"
#include "pihm_nvector.h"
#include "nv_ops.cuh"

namespace pihm_nv {

constexpr double kBigReal = DBL_MAX;

struct Scratch {
  double *partials = nullptr;   // [kPartials]
  unsigned int *ticket = nullptr;
  double *result = nullptr;     // [2] value, flag
  double *slots = nullptr;      // [2 * PIHM_NV_SLOTS] value, flag per slot
  // pinned, written by the kernels: [0..1] a reduction's value and flag, then
  // the slots' values, a device word, and the sequence number of the last
  // write (host_flag.h)
  double *host = nullptr;
  uint64_t seq = 0;
  uint64_t *seq_word() const { return (uint64_t *)(host + 2 + PIHM_NV_SLOTS + 1); }
};

// Scratch layout: partial values and flags (kMaxBlocks each, or the eight
// warps of kSeqSpread blocks for two reductions of a sequence, nv_queue.h),
// result [2], ticket, one spare, slots [2 * PIHM_NV_SLOTS].
constexpr int kSeqSpread = 128;
constexpr size_t kPartials = 16 * kSeqSpread;
static_assert(kPartials >= 2 * kMaxBlocks, "reduction partials");
constexpr size_t kScratchDoubles = kPartials + 4 + 2 * PIHM_NV_SLOTS;
constexpr size_t kHostDoubles = 2 + PIHM_NV_SLOTS + 2;

static int scratch_alloc(Scratch &s) {
  void *p = nullptr;
  if (cudaMalloc(&p, sizeof(double) * kScratchDoubles) != cudaSuccess) return -1;
  char *c = (char *)p;
  s.partials = (double *)c;
  s.result = (double *)(c + sizeof(double) * kPartials);
  s.ticket = (unsigned int *)(c + sizeof(double) * (kPartials + 2));
  s.slots = (double *)(c + sizeof(double) * (kPartials + 4));
  if (cudaMemset(p, 0, sizeof(double) * kScratchDoubles) != cudaSuccess) return -1;
  if (cudaMallocHost(&s.host, sizeof(double) * kHostDoubles) != cudaSuccess) return -1;
  std::memset(s.host, 0, sizeof(double) * kHostDoubles);
  return 0;
}

static void scratch_free(Scratch &s) {
  if (s.partials) cudaFree(s.partials);
  if (s.host) cudaFreeHost(s.host);
  s = Scratch();
}

// A vector family: the stream plus reduction scratch, shared by clones.
struct Family {
  cudaStream_t stream;
  Scratch scratch;
  int refs;
};

struct Content {
  long int length;
  int own_data;
  double *data;
  Family *fam;
};

static inline Content *C(N_Vector v) { return (Content *)v->content; }
static inline double *D(N_Vector v) { return C(v)->data; }
static inline long int L(N_Vector v) { return C(v)->length; }
static inline cudaStream_t S(N_Vector v) { return C(v)->fam->stream; }

static inline unsigned grid_for(long long n) {
  long long b = (n + kThreads - 1) / kThreads;
  if (b > 16 * 152) b = 16 * 152;
  return (unsigned)(b > 0 ? b : 1);
}

// The kernels here are programmatic dependent launches: a block waits for the
// kernel before it and reads nothing until then.  A Newton and GMRES
// iteration's fourteen operations, four of which return a value, over 31,337
// entries take 68 us instead of 86, over 3.06M 239 instead of 258.  A grid of
// one wave lets the next one's blocks in as it starts (k_red: unless its value
// stays in a slot); of more, they would hold its own blocks' places (3.06M:
// 262).
constexpr unsigned kWave = 8 * 152;  // 256-thread blocks that GB300's SMs hold at once
__device__ __forceinline__ void begin_after_previous() {
  if (gridDim.x <= kWave) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <class... P, class... A>
static int launch_after(void (*kernel)(P...), unsigned grid, unsigned block, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, kernel, P(args)...) == cudaSuccess) return 0;
  (void)cudaGetLastError();
  return -2;
}

// ---------------------------------------------------------------------------
// element-wise kernels
// ---------------------------------------------------------------------------
template <int OP>
__global__ void k_ew(long long n, double a, double b, const double *x, const double *y, double *z) {
  begin_after_previous();
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const double xv = ew_reads_x(OP) ? x[i] : 0.0;
    const double yv = ew_reads_y(OP) ? y[i] : 0.0;
    const double zv = ew_reads_z(OP) ? z[i] : 0.0;
    z[i] = ew_eval<OP>(a, b, xv, yv, zv);
  }
}

template <int OP>
static int ew(long long n, double a, double b, const double *x, const double *y, double *z,
              cudaStream_t st) {
  if (n <= 0) return 0;
  return launch_after(k_ew<OP>, grid_for(n), kThreads, st, n, a, b, x, y, z);
}

// One element-wise call after the serial N_Vector's case analysis.
static int ew_call(const EwCall<const double *> &c, long long n, cudaStream_t st) {
  double *z = const_cast<double *>(c.z);
  switch (c.op) {
    case EW_LIN: return ew<EW_LIN>(n, c.a, c.b, c.x, c.y, z, st);
    case EW_LIN1: return ew<EW_LIN1>(n, c.a, c.b, c.x, c.y, z, st);
    case EW_LIN2: return ew<EW_LIN2>(n, c.a, c.b, c.x, c.y, z, st);
    case EW_SUM: return ew<EW_SUM>(n, c.a, c.b, c.x, c.y, z, st);
    case EW_DIFF: return ew<EW_DIFF>(n, c.a, c.b, c.x, c.y, z, st);
    case EW_SCALESUM: return ew<EW_SCALESUM>(n, c.a, c.b, c.x, c.y, z, st);
    case EW_SCALEDIFF: return ew<EW_SCALEDIFF>(n, c.a, c.b, c.x, c.y, z, st);
    case EW_AXPY: return ew<EW_AXPY>(n, c.a, c.b, c.x, c.y, z, st);
    case EW_AXPY1: return ew<EW_AXPY1>(n, c.a, c.b, c.x, c.y, z, st);
    case EW_AXPYM1: return ew<EW_AXPYM1>(n, c.a, c.b, c.x, c.y, z, st);
    case EW_SCALE: return ew<EW_SCALE>(n, c.a, c.b, c.x, c.y, z, st);
    case EW_COPY: return ew<EW_COPY>(n, c.a, c.b, c.x, c.y, z, st);
    case EW_NEG: return ew<EW_NEG>(n, c.a, c.b, c.x, c.y, z, st);
    default: return -1;
  }
}

// z = a*x + b*y (cvode/src/nvec_ser/nvector_serial.c:421-506)
static int linear_sum(double a, const double *x, double b, const double *y, double *z, long long n,
                      cudaStream_t st) {
  return ew_call(select_linear_sum<const double *>(a, x, b, y, z), n, st);
}

// ---------------------------------------------------------------------------
// reductions
// ---------------------------------------------------------------------------
// x, y, w are the operands; m (optional) receives the ConstrMask output and
// z the InvTest output.
template <int OP>
__global__ void __launch_bounds__(kThreads) k_red(long long n, const double *x, const double *y, double *z,
                                                  double *partials, double *partials_f,
                                                  unsigned int *ticket, double *result,
                                                  long long wrms_n, double *host, uint64_t *host_seq,
                                                  uint64_t seq) {
  __shared__ Pair sh[kThreads / 32];
  __shared__ bool last;
  // A value left in a slot does not let the next kernel in early: behind
  // another reduction its blocks would share SMs unevenly when the places of
  // this one come free (back to back, 140,000 entries: 9.4 us, 4.6 without;
  // 20M 132 and 92).  (The wave test always holds; with it the compiler keeps
  // the loads' order that gives 99.1 us for a dot product of 20M, 103 without.)
  if (gridDim.x <= kWave && host) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  Pair acc = red_identity<OP>();
  const long long stride = (long long)gridDim.x * blockDim.x;
  long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (OP == R_DOT || OP == R_WSQ || OP == R_MAXABS || OP == R_MIN || OP == R_L1) {
    // four grid-stride entries at a time (their loads in flight together),
    // accumulated in grid-stride order
    constexpr int U = 4;
    for (; i0 < n; i0 += U * stride) {
      double xv[U], yv[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const long long i = i0 + u * stride;
        xv[u] = (i < n) ? x[i] : 0.0;
        yv[u] = (i < n && (OP == R_DOT || OP == R_WSQ)) ? y[i] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < U; u++)
        if (i0 + u * stride < n) acc = red_combine<OP>(acc, red_term<OP>(xv[u], yv[u]));
    }
  }
  for (long long i = i0; i < n; i += stride) {
    Pair t = red_identity<OP>();
    if (OP == R_DOT || OP == R_WSQ) t = red_term<OP>(x[i], y[i]);
    else if (OP == R_MAXABS || OP == R_MIN || OP == R_L1) t = red_term<OP>(x[i], 0.0);
    else if (OP == R_WSQ_MASK) {
      if (z[i] > 0.0) { double p = __dmul_rn(x[i], y[i]); t.v = __dmul_rn(p, p); }
    } else if (OP == R_INVTEST) {
      if (x[i] == 0.0) t.f = 1.0;
      else z[i] = div_rn(1.0, x[i]);
    } else if (OP == R_CONSTR) {
      // cvode/src/nvec_ser/nvector_serial.c:813-841: c = x, x = y, m = z
      const double c = x[i], v = y[i];
      double mi = 0.0;
      if (c != 0.0) {
        if (c > 1.5 || c < -1.5) {
          if (__dmul_rn(v, c) <= 0.0) { t.f = 1.0; mi = 1.0; }
        } else if (c > 0.5 || c < -0.5) {
          if (__dmul_rn(v, c) < 0.0) { t.f = 1.0; mi = 1.0; }
        }
      }
      z[i] = mi;
    } else if (OP == R_MINQ) {
      if (y[i] != 0.0) { t.v = div_rn(x[i], y[i]); t.f = 1.0; }
    }
    acc = red_combine<OP>(acc, t);
  }
  acc = red_block<OP>(acc, sh);
  if (threadIdx.x == 0) {
    partials[blockIdx.x] = acc.v;
    partials_f[blockIdx.x] = acc.f;
    __threadfence();
    const unsigned int t = atomicAdd(ticket, 1u);
    last = (t == gridDim.x - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  // the last block combines the partials in a fixed order
  Pair v = red_identity<OP>();
  for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x) {
    Pair q = {((volatile double *)partials)[b], ((volatile double *)partials_f)[b]};
    v = red_combine<OP>(v, q);
  }
  v = red_block<OP>(v, sh);
  if (threadIdx.x == 0) {
    // wrms_n > 0: the WRMS norm sqrt(sum / n) itself, as N_VWrmsNorm forms it
    result[0] = wrms_n > 0 ? __dsqrt_rn(__ddiv_rn(v.v, (double)wrms_n)) : v.v;
    result[1] = v.f;
    *ticket = 0u;
    if (host) {
      host[0] = result[0];
      host[1] = v.f;
      pihm::host_flag_set(host_seq, seq);
    }
  }
}

// slots 0..count-1 and a device word to the host
__global__ void k_fetch(const double *slots, int count, const unsigned int *word, double *host, uint64_t *host_seq,
                        uint64_t seq) {
  if ((int)threadIdx.x < count) host[2 + threadIdx.x] = slots[2 * threadIdx.x];
  if (threadIdx.x == 0 && word) *(unsigned int *)(host + 2 + PIHM_NV_SLOTS) = *word;
  __threadfence_system();
  __syncwarp();
  if (threadIdx.x == 0) pihm::host_flag_set(host_seq, seq);
}

// z = a*x + b*y with a and b formed from device-resident slots: one thread
// of each block forms the coefficients and makes the serial N_Vector's case
// analysis from their values (operand tags 0 = x, 1 = y; ztag 0 when z is x,
// 1 when z is y, 2 otherwise), then the block runs the chosen variant.
template <int OP>
__device__ __forceinline__ void ew_loop(long long n, double a, double b, const double *x, const double *y,
                                        double *z) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const double xv = ew_reads_x(OP) ? x[i] : 0.0;
    const double yv = ew_reads_y(OP) ? y[i] : 0.0;
    const double zv = ew_reads_z(OP) ? z[i] : 0.0;
    z[i] = ew_eval<OP>(a, b, xv, yv, zv);
  }
}

__global__ void k_lin_coef(long long n, int ka, int sa, double va, int kb, int sb, double vb, int ztag,
                           const double *x, const double *y, double *z, const double *slots) {
  __shared__ int s_op, s_xt, s_yt;
  __shared__ double s_a, s_b;
  begin_after_previous();
  if (threadIdx.x == 0) {
    const double a = coef_value(ka, va, ka == COEF_HOST ? 0.0 : slots[2 * sa]);
    const double b = coef_value(kb, vb, kb == COEF_HOST ? 0.0 : slots[2 * sb]);
    const EwCall<int> c = select_linear_sum<int>(a, 0, b, 1, ztag);
    s_op = c.op;
    s_a = c.a;
    s_b = c.b;
    s_xt = c.x;
    s_yt = c.y;
  }
  __syncthreads();
  const double *px = s_xt == 0 ? x : y, *py = s_yt == 0 ? x : y;
  const double a = s_a, b = s_b;
  switch (s_op) {
    case EW_LIN: ew_loop<EW_LIN>(n, a, b, px, py, z); break;
    case EW_LIN1: ew_loop<EW_LIN1>(n, a, b, px, py, z); break;
    case EW_LIN2: ew_loop<EW_LIN2>(n, a, b, px, py, z); break;
    case EW_SUM: ew_loop<EW_SUM>(n, a, b, px, py, z); break;
    case EW_DIFF: ew_loop<EW_DIFF>(n, a, b, px, py, z); break;
    case EW_SCALESUM: ew_loop<EW_SCALESUM>(n, a, b, px, py, z); break;
    case EW_SCALEDIFF: ew_loop<EW_SCALEDIFF>(n, a, b, px, py, z); break;
    case EW_AXPY: ew_loop<EW_AXPY>(n, a, b, px, py, z); break;
    case EW_AXPY1: ew_loop<EW_AXPY1>(n, a, b, px, py, z); break;
    default: ew_loop<EW_AXPYM1>(n, a, b, px, py, z); break;
  }
}

}  // namespace pihm_nv

namespace pihm_nv {

// Launch a reduction into `scratch` (partials [kMaxBlocks] then flags [kMaxBlocks]
// carved from the caller's buffer), leave the result in result_dev[0..1].
template <int OP>
static int red_launch(long long n, const double *x, const double *y, double *z, double *partials,
                      unsigned int *ticket, double *result_dev, cudaStream_t st, long long wrms_n = 0,
                      double *host = nullptr, uint64_t *host_seq = nullptr, uint64_t seq = 0) {
  const unsigned g = red_grid_for(n);
  return launch_after(k_red<OP>, g, kThreads, st, n, x, y, z, partials, partials + kMaxBlocks, ticket, result_dev,
                      wrms_n, host, host_seq, seq);
}

template <int OP>
static int red_family(Family *f, long long n, const double *x, const double *y, double *z, double out[2]) {
  Scratch &s = f->scratch;
  const uint64_t seq = ++s.seq;
  if (red_launch<OP>(n, x, y, z, s.partials, s.ticket, s.result, f->stream, 0, s.host, s.seq_word(), seq)) return -2;
  if (!pihm::host_flag_wait(s.seq_word(), seq, f->stream)) return -2;
  out[0] = s.host[0];
  out[1] = s.host[1];
  return 0;
}

// ---------------------------------------------------------------------------
// sequences: element-wise operations and the reduction that ends them
// ---------------------------------------------------------------------------
// r = OP(a, b, x, y, z) for a run-time operation code
template <int U>
__device__ __forceinline__ void seq_eval(int op, double a, double b, const double (&x)[U], const double (&y)[U],
                                         const double (&z)[U], double (&r)[U]) {
#define PIHM_SEQ_CASE(OP)                                                  \
  case OP:                                                                 \
    _Pragma("unroll") for (int u = 0; u < U; u++) r[u] = ew_eval<OP>(a, b, x[u], y[u], z[u]); \
    break;
  switch (op) {
    PIHM_SEQ_CASE(EW_LIN)
    PIHM_SEQ_CASE(EW_LIN1)
    PIHM_SEQ_CASE(EW_LIN2)
    PIHM_SEQ_CASE(EW_SUM)
    PIHM_SEQ_CASE(EW_DIFF)
    PIHM_SEQ_CASE(EW_SCALESUM)
    PIHM_SEQ_CASE(EW_SCALEDIFF)
    PIHM_SEQ_CASE(EW_AXPY)
    PIHM_SEQ_CASE(EW_AXPY1)
    PIHM_SEQ_CASE(EW_AXPYM1)
    PIHM_SEQ_CASE(EW_CONST)
    PIHM_SEQ_CASE(EW_PROD)
    PIHM_SEQ_CASE(EW_DIV)
    PIHM_SEQ_CASE(EW_SCALE)
    PIHM_SEQ_CASE(EW_COPY)
    PIHM_SEQ_CASE(EW_NEG)
    PIHM_SEQ_CASE(EW_ABS)
    PIHM_SEQ_CASE(EW_INV)
    PIHM_SEQ_CASE(EW_ADDCONST)
    default: break;
  }
#undef PIHM_SEQ_CASE
}

// An operation as a block runs it: coefficients from slots resolved.
struct SeqHead {
  double a, b;
  const double *x, *y;
  double *z;
  int op, fwd;
};

template <int U>
__device__ __forceinline__ void seq_load(const SeqHead &h, const long long (&i)[U], const bool (&on)[U],
                                         const double (&prev)[U], double (&x)[U], double (&y)[U], double (&z)[U]) {
  const bool lx = ew_reads_x(h.op) && !(h.fwd & SEQ_X), ly = ew_reads_y(h.op) && !(h.fwd & SEQ_Y),
             lz = ew_reads_z(h.op) && !(h.fwd & SEQ_Z);
  __builtin_assume(__isGlobal(h.x));
  __builtin_assume(__isGlobal(h.y));
  __builtin_assume(__isGlobal(h.z));
#pragma unroll
  for (int u = 0; u < U; u++) {
    x[u] = lx && on[u] ? h.x[i[u]] : prev[u];
    y[u] = ly && on[u] ? h.y[i[u]] : prev[u];
    z[u] = lz && on[u] ? h.z[i[u]] : prev[u];
  }
}

// One reduction within a block of k_seq.  kSpread: `part` has a value per
// warp of the reduction order.
template <int RED, bool kSpread, int kT>
__device__ __forceinline__ void seq_tail_block(double acc, int vwarp, bool writer, double *part, double *sh) {
  const double v = warp_tree<RED>(acc);
  if (writer) {
    if (kSpread) part[vwarp] = v;
    else sh[threadIdx.x >> 5] = v;
  }
}
// A sequence over a vector: element-wise operations in order, then nothing
// (RA < 0), one reduction (RA) or two (RA, RB).  An operation on a vector the
// one before wrote takes the value from registers, and a result that is
// overwritten unread is not stored.
//
// What it saves: a separate kernel costs about 4 us an operation in front of
// a reduction (four operations and a dot product over 6,200 entries: 27.4 us
// until the value is on the host, 12.9 here; a dot product alone 11.5, an
// empty kernel 7.0), and each passes over the vectors.
//
// kSpread (short vectors, one pass): a warp has one FP64 instruction in
// flight, 69 clocks, whatever its threads do beside it, and an SM takes one
// every 20, so work is spread over warps rather than over a thread's
// registers.  The four entries a thread of the reduction order accumulates go
// to four warps of a block, one per scheduler, and a block carries one warp
// of that order, whose tree's value it leaves in partials[8 * block + warp];
// the last block finishes the trees of the order's blocks.  Eight linear sums
// and a dot product over 6,200 entries: 13.7 us, with four entries a thread
// 18.0.  Long vectors fill the SMs with four entries a thread (k_red's
// layout) and are bound by the FP64 pipe; the spread form's tail grows with
// the blocks (eight operations and a dot product, spread / four a thread:
// 17.4 / 21.5 us over 90,000 entries, 22.3 / 21.3 over 150,000).
template <int RA, int RB, bool kSpread, int kT>
__global__ void __launch_bounds__(kT, 4) k_seq(const __grid_constant__ Seq q) {
  constexpr int R0 = RA < 0 ? 0 : RA, R1 = RB < 0 ? 0 : RB, U = kSpread ? 1 : 4;
  __shared__ SeqHead s_op[kSeqOps];
  __shared__ double sh[2][8];
  __shared__ double s_term[kSpread ? 2 : 1][kSpread ? kT : 1];
  __shared__ bool last;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const long long n = q.n;
  const int nblk = (int)red_grid_for(n);
  const long long stride = (long long)nblk * kThreads;
  begin_after_previous();
  if (tid < q.nops) {
    const SeqOp &o = q.op[tid];
    SeqHead h = {o.a, o.b, o.x, o.y, o.z, o.code, o.fwd};
    if (o.code == EW_COUNT) {
      const double a = coef_value(o.ka, o.a, o.ka == COEF_HOST ? 0.0 : q.slots[2 * o.sa]);
      const double b = coef_value(o.kb, o.b, o.kb == COEF_HOST ? 0.0 : q.slots[2 * o.sb]);
      const EwCall<int> c = select_linear_sum<int>(a, 0, b, 1, o.ztag);
      const int fx = (o.fwd & SEQ_X) ? 1 : 0, fy = (o.fwd & SEQ_Y) ? 1 : 0;
      h.op = c.op;
      h.a = c.a;
      h.b = c.b;
      h.x = c.x == 0 ? o.x : o.y;
      h.y = c.y == 0 ? o.x : o.y;
      h.fwd = (o.fwd & (SEQ_Z | SEQ_DEAD)) | ((c.x == 0 ? fx : fy) ? SEQ_X : 0) | ((c.y == 0 ? fx : fy) ? SEQ_Y : 0);
    }
    s_op[tid] = h;
  }
  __syncthreads();
  Pair acc[2] = {red_identity<R0>(), red_identity<R1>()};
  const int nops = q.nops;
  const int vwarp = kSpread ? blockIdx.x : blockIdx.x * (kT / 32) + wid;
  for (long long i0 = (long long)vwarp * 32 + lane + (kSpread ? wid * stride : 0); i0 < n; i0 += 4 * stride) {
    double prev[U], x[U], y[U], z[U];
    long long i[U];
    bool on[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      prev[u] = 0.0;
      i[u] = i0 + u * stride;
      on[u] = i[u] < n;
    }
    for (int p = 0; p < nops; p++) {
      const SeqHead h = s_op[p];
      seq_load<U>(h, i, on, prev, x, y, z);
      seq_eval<U>(h.op, h.a, h.b, x, y, z, prev);
      if (!(h.fwd & SEQ_DEAD)) {
#pragma unroll
        for (int u = 0; u < U; u++)
          if (on[u]) h.z[i[u]] = prev[u];
      }
    }
#pragma unroll
    for (int r = 0; r < (RA < 0 ? 0 : (RB < 0 ? 1 : 2)); r++) {
      const SeqRed &d = q.red[r];
      const bool two = (r == 0 ? R0 : R1) == R_DOT || (r == 0 ? R0 : R1) == R_WSQ;
      Pair t[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        x[u] = (d.fwd & SEQ_X) || !on[u] ? prev[u] : d.x[i[u]];
        y[u] = !two ? 0.0 : ((d.fwd & SEQ_Y) || !on[u] ? prev[u] : d.y[i[u]]);
      }
#pragma unroll
      for (int u = 0; u < U; u++) t[u] = r == 0 ? red_term<R0>(x[u], y[u]) : red_term<R1>(x[u], y[u]);
#pragma unroll
      for (int u = 0; u < U; u++) {
        if (kSpread) s_term[r][tid] = t[u].v;
        else if (on[u]) acc[r] = r == 0 ? red_combine<R0>(acc[r], t[u]) : red_combine<R1>(acc[r], t[u]);
      }
    }
  }
  if (RA < 0) return;

  double *part[2] = {q.partials, q.partials + (kSpread ? 8 * kSeqSpread : kMaxBlocks)};
  if (kSpread) {
    __syncthreads();
    // the second reduction's warps follow the first's
    const int r = wid;
    if (wid < (RB < 0 ? 1 : 2)) {
      const long long i0 = (long long)vwarp * 32 + lane;
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (i0 + u * stride < n) {
          const Pair t = {s_term[RB < 0 ? 0 : r][u * 32 + lane], 0.0};
          if (u == 0) acc[0] = r == 0 ? red_first<R0>(t) : red_first<R1>(t);
          else acc[0] = r == 0 ? red_combine<R0>(acc[0], t) : red_combine<R1>(acc[0], t);
        }
      if (r == 0) seq_tail_block<R0, true, kT>(acc[0].v, vwarp, lane == 0, part[0], sh[0]);
      else seq_tail_block<R1, true, kT>(i0 < n ? acc[0].v : red_identity<R1>().v, vwarp, lane == 0, part[1], sh[1]);
    }
  } else {
    seq_tail_block<R0, false, kT>(acc[0].v, vwarp, lane == 0, part[0], sh[0]);
    if (RB >= 0) seq_tail_block<R1, false, kT>(acc[1].v, vwarp, lane == 0, part[1], sh[1]);
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    if (!kSpread) {
      part[0][blockIdx.x] = eight_tree<R0>(sh[0]);
      if (RB >= 0) part[1][blockIdx.x] = eight_tree<R1>(sh[1]);
      __threadfence();
    }
    last = atomicAdd(q.ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  // the last block combines the blocks' values in a fixed order
  tree_last<R0, kSpread, kT>(nblk, part[0], sh[0]);
  if (RB >= 0) tree_last<R1, kSpread, kT>(nblk, part[1], sh[1]);
  __syncthreads();
  if (wid == 0 && lane < (RB < 0 ? 1 : 2)) {
    const SeqRed &d = q.red[lane];
    double v = lane == 0 ? eight_tree<R0>(sh[0]) : eight_tree<R1>(sh[1]);
    // the WRMS norm itself, sqrt(sum / n), as N_VWrmsNorm forms it
    if (d.wrms_n > 0) v = __dsqrt_rn(__ddiv_rn(v, (double)d.wrms_n));
    d.out[0] = v;
    d.out[1] = 0.0;
    if (q.host_seq) q.host[lane] = v;
  }
  if (tid == 0) *q.ticket = 0u;
  if (q.host_seq == nullptr) return;
  __syncthreads();
  for (int k = tid; k < q.fetch; k += kT) q.host[2 + k] = ((const volatile double *)q.slots)[2 * k];
  if (tid == 0 && q.word) *(unsigned int *)(q.host + 2 + PIHM_NV_SLOTS) = *q.word;
  __threadfence_system();
  __syncthreads();
  if (tid == 0) pihm::host_flag_set(q.host_seq, q.seq);
}

template <int RA, int RB, bool kSpread, int kT>
static int seq_launch_t(const Seq &q, unsigned grid, cudaStream_t st) {
  return launch_after(k_seq<RA, RB, kSpread, kT>, grid, kT, st, q);
}

template <int RA, int RB>
static int seq_launch_r(const Seq &q, cudaStream_t st) {
  // 131,072 entries and fewer spread: see k_seq
  const unsigned g = red_grid_for(q.n);
  if (g <= kSeqSpread) return seq_launch_t<RA, RB, true, 128>(q, g * (kThreads / 32), st);
  return seq_launch_t<RA, RB, false, kThreads>(q, g, st);
}

static int seq_launch(const Seq &q, cudaStream_t st) {
  switch (q.nred ? q.red[0].op : -1) {
    case R_DOT: return q.nred == 2 ? seq_launch_r<R_DOT, R_DOT>(q, st) : seq_launch_r<R_DOT, -1>(q, st);
    case R_WSQ: return seq_launch_r<R_WSQ, -1>(q, st);
    case R_MAXABS: return seq_launch_r<R_MAXABS, -1>(q, st);
    case R_MIN: return q.nred == 2 ? seq_launch_r<R_MIN, R_WSQ>(q, st) : seq_launch_r<R_MIN, -1>(q, st);
    default: return seq_launch_r<-1, -1>(q, st);
  }
}

}  // namespace pihm_nv

using namespace pihm_nv;

extern "C" {

static N_Vector new_empty(Family *fam);

static struct _generic_N_Vector_Ops *make_ops() {
  struct _generic_N_Vector_Ops *o = (struct _generic_N_Vector_Ops *)calloc(1, sizeof(*o));
  o->nvgetvectorid = N_VGetVectorID_PihmGpu;
  o->nvclone = N_VClone_PihmGpu;
  o->nvcloneempty = N_VCloneEmpty_PihmGpu;
  o->nvdestroy = N_VDestroy_PihmGpu;
  o->nvspace = N_VSpace_PihmGpu;
  o->nvgetarraypointer = N_VGetArrayPointer_PihmGpu;
  o->nvsetarraypointer = N_VSetArrayPointer_PihmGpu;
  o->nvlinearsum = N_VLinearSum_PihmGpu;
  o->nvconst = N_VConst_PihmGpu;
  o->nvprod = N_VProd_PihmGpu;
  o->nvdiv = N_VDiv_PihmGpu;
  o->nvscale = N_VScale_PihmGpu;
  o->nvabs = N_VAbs_PihmGpu;
  o->nvinv = N_VInv_PihmGpu;
  o->nvaddconst = N_VAddConst_PihmGpu;
  o->nvdotprod = N_VDotProd_PihmGpu;
  o->nvmaxnorm = N_VMaxNorm_PihmGpu;
  o->nvwrmsnorm = N_VWrmsNorm_PihmGpu;
  o->nvwrmsnormmask = N_VWrmsNormMask_PihmGpu;
  o->nvmin = N_VMin_PihmGpu;
  o->nvwl2norm = N_VWL2Norm_PihmGpu;
  o->nvl1norm = N_VL1Norm_PihmGpu;
  o->nvcompare = N_VCompare_PihmGpu;
  o->nvinvtest = N_VInvTest_PihmGpu;
  o->nvconstrmask = N_VConstrMask_PihmGpu;
  o->nvminquotient = N_VMinQuotient_PihmGpu;
  return o;
}

static N_Vector new_empty(Family *fam) {
  N_Vector v = (N_Vector)calloc(1, sizeof(*v));
  Content *c = (Content *)calloc(1, sizeof(Content));
  if (!v || !c) {
    free(v);
    free(c);
    return nullptr;
  }
  v->ops = make_ops();
  v->content = c;
  c->fam = fam;
  fam->refs++;
  return v;
}

static Family *new_family(void *stream) {
  Family *f = new Family();
  f->stream = (cudaStream_t)stream;
  f->refs = 0;
  if (scratch_alloc(f->scratch)) {
    scratch_free(f->scratch);
    delete f;
    return nullptr;
  }
  return f;
}

N_Vector N_VNew_PihmGpu(long int length, void *stream) {
  if (length < 0) return nullptr;
  Family *f = new_family(stream);
  if (!f) return nullptr;
  N_Vector v = new_empty(f);
  if (!v) return nullptr;
  Content *c = C(v);
  c->length = length;
  c->own_data = 1;
  if (length > 0 && cudaMalloc(&c->data, sizeof(double) * length) != cudaSuccess) {
    N_VDestroy_PihmGpu(v);
    return nullptr;
  }
  return v;
}

N_Vector N_VMake_PihmGpu(long int length, double *dev_data, void *stream) {
  if (length < 0) return nullptr;
  Family *f = new_family(stream);
  if (!f) return nullptr;
  N_Vector v = new_empty(f);
  if (!v) return nullptr;
  C(v)->length = length;
  C(v)->own_data = 0;
  C(v)->data = dev_data;
  return v;
}

double *N_VGetDeviceArrayPointer_PihmGpu(N_Vector v) { return D(v); }
long int N_VGetLength_PihmGpu(N_Vector v) { return L(v); }

int N_VCopyFromHost_PihmGpu(N_Vector v, const double *host) {
  if (cudaMemcpyAsync(D(v), host, sizeof(double) * L(v), cudaMemcpyHostToDevice, S(v)) != cudaSuccess) return -2;
  return cudaStreamSynchronize(S(v)) == cudaSuccess ? 0 : -2;
}

int N_VCopyToHost_PihmGpu(N_Vector v, double *host) {
  if (cudaMemcpyAsync(host, D(v), sizeof(double) * L(v), cudaMemcpyDeviceToHost, S(v)) != cudaSuccess) return -2;
  return cudaStreamSynchronize(S(v)) == cudaSuccess ? 0 : -2;
}

N_Vector_ID N_VGetVectorID_PihmGpu(N_Vector v) {
  (void)v;
  return SUNDIALS_NVEC_CUSTOM;
}

N_Vector N_VCloneEmpty_PihmGpu(N_Vector w) {
  N_Vector v = new_empty(C(w)->fam);
  if (!v) return nullptr;
  C(v)->length = L(w);
  C(v)->own_data = 0;
  C(v)->data = nullptr;
  return v;
}

N_Vector N_VClone_PihmGpu(N_Vector w) {
  N_Vector v = N_VCloneEmpty_PihmGpu(w);
  if (!v) return nullptr;
  if (L(w) > 0) {
    if (cudaMalloc(&C(v)->data, sizeof(double) * L(w)) != cudaSuccess) {
      N_VDestroy_PihmGpu(v);
      return nullptr;
    }
    C(v)->own_data = 1;
  }
  return v;
}

void N_VDestroy_PihmGpu(N_Vector v) {
  if (!v) return;
  Content *c = C(v);
  if (c) {
    if (c->own_data && c->data) cudaFree(c->data);
    Family *f = c->fam;
    if (f && --f->refs == 0) {
      scratch_free(f->scratch);
      delete f;
    }
    free(c);
  }
  free(v->ops);
  free(v);
}

void N_VSpace_PihmGpu(N_Vector v, long int *lrw, long int *liw) {
  *lrw = L(v);
  *liw = 1;
}

double *N_VGetArrayPointer_PihmGpu(N_Vector v) { return D(v); }
void N_VSetArrayPointer_PihmGpu(double *v_data, N_Vector v) {
  if (L(v) > 0) C(v)->data = v_data;
}

void N_VLinearSum_PihmGpu(double a, N_Vector x, double b, N_Vector y, N_Vector z) {
  linear_sum(a, D(x), b, D(y), D(z), L(x), S(z));
}
void N_VConst_PihmGpu(double c, N_Vector z) { ew<EW_CONST>(L(z), c, 0, nullptr, nullptr, D(z), S(z)); }
void N_VProd_PihmGpu(N_Vector x, N_Vector y, N_Vector z) { ew<EW_PROD>(L(x), 0, 0, D(x), D(y), D(z), S(z)); }
void N_VDiv_PihmGpu(N_Vector x, N_Vector y, N_Vector z) { ew<EW_DIV>(L(x), 0, 0, D(x), D(y), D(z), S(z)); }
void N_VScale_PihmGpu(double c, N_Vector x, N_Vector z) {
  // cvode/src/nvec_ser/nvector_serial.c:559-584
  ew_call(select_scale<const double *>(c, D(x), D(z)), L(x), S(z));
}
void N_VAbs_PihmGpu(N_Vector x, N_Vector z) { ew<EW_ABS>(L(x), 0, 0, D(x), nullptr, D(z), S(z)); }
void N_VInv_PihmGpu(N_Vector x, N_Vector z) { ew<EW_INV>(L(x), 0, 0, D(x), nullptr, D(z), S(z)); }
void N_VAddConst_PihmGpu(N_Vector x, double b, N_Vector z) {
  ew<EW_ADDCONST>(L(x), 0, b, D(x), nullptr, D(z), S(z));
}
void N_VCompare_PihmGpu(double c, N_Vector x, N_Vector z) {
  ew<EW_COMPARE>(L(x), c, 0, D(x), nullptr, D(z), S(z));
}

double N_VDotProd_PihmGpu(N_Vector x, N_Vector y) {
  double r[2] = {NAN, 0};
  red_family<R_DOT>(C(x)->fam, L(x), D(x), D(y), nullptr, r);
  return r[0];
}
double N_VMaxNorm_PihmGpu(N_Vector x) {
  double r[2] = {NAN, 0};
  red_family<R_MAXABS>(C(x)->fam, L(x), D(x), nullptr, nullptr, r);
  return r[0];
}
double N_VWrmsNorm_PihmGpu(N_Vector x, N_Vector w) {
  double r[2] = {NAN, 0};
  red_family<R_WSQ>(C(x)->fam, L(x), D(x), D(w), nullptr, r);
  return sqrt(r[0] / (double)L(x));
}
double N_VWrmsNormMask_PihmGpu(N_Vector x, N_Vector w, N_Vector id) {
  double r[2] = {NAN, 0};
  red_family<R_WSQ_MASK>(C(x)->fam, L(x), D(x), D(w), D(id), r);
  return sqrt(r[0] / (double)L(x));
}
double N_VMin_PihmGpu(N_Vector x) {
  double r[2] = {NAN, 0};
  red_family<R_MIN>(C(x)->fam, L(x), D(x), nullptr, nullptr, r);
  return r[0];
}
double N_VWL2Norm_PihmGpu(N_Vector x, N_Vector w) {
  double r[2] = {NAN, 0};
  red_family<R_WSQ>(C(x)->fam, L(x), D(x), D(w), nullptr, r);
  return sqrt(r[0]);
}
double N_VL1Norm_PihmGpu(N_Vector x) {
  double r[2] = {NAN, 0};
  red_family<R_L1>(C(x)->fam, L(x), D(x), nullptr, nullptr, r);
  return r[0];
}
int N_VInvTest_PihmGpu(N_Vector x, N_Vector z) {
  double r[2] = {0, 1};
  red_family<R_INVTEST>(C(x)->fam, L(x), D(x), nullptr, D(z), r);
  return r[1] == 0.0;
}
int N_VConstrMask_PihmGpu(N_Vector c, N_Vector x, N_Vector m) {
  double r[2] = {0, 1};
  red_family<R_CONSTR>(C(x)->fam, L(x), D(c), D(x), D(m), r);
  return r[1] == 0.0;
}
double N_VMinQuotient_PihmGpu(N_Vector num, N_Vector denom) {
  double r[2] = {NAN, 0};
  red_family<R_MINQ>(C(num)->fam, L(num), D(num), D(denom), nullptr, r);
  return (r[1] != 0.0) ? r[0] : kBigReal;
}

// ---------------------------------------------------------------------------
// device-resident scalars
// ---------------------------------------------------------------------------
int N_VDotProdSlot_PihmGpu(N_Vector x, N_Vector y, int slot) {
  if (!x || !y || slot < 0 || slot >= PIHM_NV_SLOTS) return -1;
  Scratch &s = C(x)->fam->scratch;
  return red_launch<R_DOT>(L(x), D(x), D(y), nullptr, s.partials, s.ticket, s.slots + 2 * slot, S(x));
}

int N_VWrmsNormSlot_PihmGpu(N_Vector x, N_Vector w, int slot) {
  if (!x || !w || slot < 0 || slot >= PIHM_NV_SLOTS || L(x) <= 0) return -1;
  Scratch &s = C(x)->fam->scratch;
  return red_launch<R_WSQ>(L(x), D(x), D(w), nullptr, s.partials, s.ticket, s.slots + 2 * slot, S(x), L(x));
}

int N_VLinearSumCoef_PihmGpu(const pihm_nv_coef *a, N_Vector x, const pihm_nv_coef *b, N_Vector y,
                             N_Vector z) {
  if (!a || !b || !x || !y || !z) return -1;
  for (const pihm_nv_coef *c : {a, b})
    if (c->kind < PIHM_NV_COEF_HOST || c->kind > PIHM_NV_COEF_NEG_INV_INV ||
        (c->kind != PIHM_NV_COEF_HOST && (c->slot < 0 || c->slot >= PIHM_NV_SLOTS)))
      return -1;
  const long long n = L(x);
  if (a->kind == PIHM_NV_COEF_HOST && b->kind == PIHM_NV_COEF_HOST)
    return linear_sum(a->value, D(x), b->value, D(y), D(z), n, S(z));
  if (n <= 0) return 0;
  const int ztag = D(z) == D(x) ? 0 : (D(z) == D(y) ? 1 : 2);
  return launch_after(k_lin_coef, grid_for(n), kThreads, S(z), n, a->kind, a->slot, a->value, b->kind, b->slot,
                      b->value, ztag, D(x), D(y), D(z), C(z)->fam->scratch.slots);
}

int N_VFetchSlots_PihmGpu(N_Vector v, int count, double *out, const unsigned int *dev_word,
                          unsigned int *word_out) {
  if (!v || count < 0 || count > PIHM_NV_SLOTS || (count > 0 && !out) || (dev_word && !word_out)) return -1;
  Scratch &s = C(v)->fam->scratch;
  const uint64_t seq = ++s.seq;
  k_fetch<<<1, 32, 0, S(v)>>>(s.slots, count, dev_word, s.host, s.seq_word(), seq);
  if (cudaGetLastError() != cudaSuccess || !pihm::host_flag_wait(s.seq_word(), seq, S(v))) return -2;
  for (int i = 0; i < count; i++) out[i] = s.host[2 + i];
  if (dev_word) *word_out = *(const unsigned int *)(s.host + 2 + PIHM_NV_SLOTS);
  return 0;
}

void *N_VGetStream_PihmGpu(N_Vector v) { return v ? (void *)S(v) : nullptr; }

// ---------------------------------------------------------------------------
// raw-pointer entry points: a library workspace per stream, created on first
// use and kept until the process exits
// ---------------------------------------------------------------------------
static std::mutex g_ws_mu;
static std::map<cudaStream_t, Family *> g_ws;

static Family *stream_family(void *stream) {
  std::lock_guard<std::mutex> lk(g_ws_mu);
  auto it = g_ws.find((cudaStream_t)stream);
  if (it != g_ws.end()) return it->second;
  Family *f = new_family(stream);
  if (f) g_ws[(cudaStream_t)stream] = f;
  return f;
}

int pihm_gpu_nv_linear_sum(double a, const double *x, double b, const double *y, double *z, int64_t n,
                           void *stream) {
  if (n < 0 || (n > 0 && (!x || !y || !z))) return -1;
  return linear_sum(a, x, b, y, z, n, (cudaStream_t)stream);
}

int pihm_gpu_nv_wrms_norm(const double *x, const double *w, int64_t n, void *stream, double *result) {
  if (n <= 0 || !x || !w || !result) return -1;
  Family *f = stream_family(stream);
  if (!f) return -5;
  double r[2];
  if (red_family<R_WSQ>(f, n, x, w, nullptr, r)) return -2;
  *result = sqrt(r[0] / (double)n);
  return 0;
}

int pihm_gpu_nv_dot_prod(const double *x, const double *y, int64_t n, void *stream, double *result) {
  if (n <= 0 || !x || !y || !result) return -1;
  Family *f = stream_family(stream);
  if (!f) return -5;
  double r[2];
  if (red_family<R_DOT>(f, n, x, y, nullptr, r)) return -2;
  *result = r[0];
  return 0;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// the queue (nv_queue.h)
// ---------------------------------------------------------------------------
namespace pihm_nv {

// whether the vectors (null: not an operand) are the queue's, adopting z's
// family and length when nothing is queued
bool NvQueue::take(N_Vector z, N_Vector x, N_Vector y) {
  if (z->ops->nvgetvectorid != N_VGetVectorID_PihmGpu || L(z) <= 0) return false;
  if (empty()) {
    fam = C(z)->fam;
    q.n = L(z);
  }
  for (N_Vector v : {z, x, y})
    if (v && (v->ops->nvgetvectorid != N_VGetVectorID_PihmGpu || C(v)->fam != fam || L(v) != q.n)) return false;
  return true;
}

void NvQueue::push(const SeqOp &o) {
  if (q.nred > 0 || q.nops == kSeqOps) {
    flush();
  }
  SeqOp &d = q.op[q.nops];
  d = o;
  if (q.nops > 0) {
    const double *pz = q.op[q.nops - 1].z;
    d.fwd = (uint8_t)((o.x == pz ? SEQ_X : 0) | (o.y == pz ? SEQ_Y : 0) | (o.z == pz ? SEQ_Z : 0));
  }
  q.nops++;
}

void NvQueue::push_red(const SeqRed &r) {
  if (q.nred == 2 || (q.nred == 1 && !(q.red[0].op == R_DOT && r.op == R_DOT) &&
                      !(q.red[0].op == R_MIN && r.op == R_WSQ))) {
    flush();
  }
  SeqRed &d = q.red[q.nred++];
  d = r;
  if (q.nops > 0) {
    const double *pz = q.op[q.nops - 1].z;
    d.fwd = (uint8_t)((r.x == pz ? SEQ_X : 0) | (r.y == pz ? SEQ_Y : 0));
  }
}

int NvQueue::launch(bool back, int fetch, const unsigned int *word) {
  // results that nothing reads before they are overwritten
  for (int p = 0; p < q.nops; p++) {
    const double *z = q.op[p].z;
    for (int r = p + 1; r < q.nops; r++) {
      const SeqOp &o = q.op[r];
      const bool sum = o.code == EW_COUNT, prev = r == p + 1;
      if (!prev && (((sum || ew_reads_x(o.code)) && o.x == z) || ((sum || ew_reads_y(o.code)) && o.y == z) ||
                    ((sum || ew_reads_z(o.code)) && o.z == z)))
        break;
      if (o.z == z) {
        q.op[p].fwd |= SEQ_DEAD;
        break;
      }
    }
  }
  Scratch &s = fam->scratch;
  q.partials = s.partials;
  q.slots = s.slots;
  q.ticket = s.ticket;
  q.host = s.host;
  q.host_seq = back ? s.seq_word() : nullptr;
  q.seq = back ? ++s.seq : 0;
  q.fetch = fetch;
  q.word = word;
  if (seq_launch(q, fam->stream) || (back && !pihm::host_flag_wait(s.seq_word(), s.seq, fam->stream))) failed = true;
  q.nops = q.nred = 0;
  return failed ? -2 : 0;
}

int NvQueue::flush() {
  return empty() ? 0 : launch(false);
}

bool NvQueue::linear_sum(double a, N_Vector x, double b, N_Vector y, N_Vector z) {
  if (z->ops->nvlinearsum != N_VLinearSum_PihmGpu || !take(z, x, y)) return false;
  const EwCall<const double *> c = select_linear_sum<const double *>(a, D(x), b, D(y), D(z));
  push({c.x, c.y, D(z), c.a, c.b, (uint8_t)c.op});
  return true;
}

bool NvQueue::linear_sum_coef(const pihm_nv_coef &a, N_Vector x, const pihm_nv_coef &b, N_Vector y, N_Vector z) {
  if (a.kind == PIHM_NV_COEF_HOST && b.kind == PIHM_NV_COEF_HOST) return linear_sum(a.value, x, b.value, y, z);
  if (!take(z, x, y)) return false;
  const uint8_t ztag = D(z) == D(x) ? 0 : (D(z) == D(y) ? 1 : 2);
  push({D(x), D(y), D(z), a.value, b.value, EW_COUNT, 0, (uint8_t)a.kind, (uint8_t)a.slot, (uint8_t)b.kind,
        (uint8_t)b.slot, ztag});
  return true;
}

bool NvQueue::scale(double c, N_Vector x, N_Vector z) {
  if (z->ops->nvscale != N_VScale_PihmGpu || !take(z, x, nullptr)) return false;
  const EwCall<const double *> e = select_scale<const double *>(c, D(x), D(z));
  push({e.x, e.x, D(z), e.a, e.b, (uint8_t)e.op});
  return true;
}

bool NvQueue::ew(int op, double a, double b, N_Vector x, N_Vector y, N_Vector z) {
  const _generic_N_Vector_Ops *o = z->ops;
  bool own = false;
  switch (op) {
    case EW_CONST: own = o->nvconst == N_VConst_PihmGpu; break;
    case EW_ABS: own = o->nvabs == N_VAbs_PihmGpu; break;
    case EW_INV: own = o->nvinv == N_VInv_PihmGpu; break;
    case EW_DIV: own = o->nvdiv == N_VDiv_PihmGpu; break;
    case EW_PROD: own = o->nvprod == N_VProd_PihmGpu; break;
    case EW_ADDCONST: own = o->nvaddconst == N_VAddConst_PihmGpu; break;
    default: break;
  }
  if (!own || !take(z, x, y)) return false;
  push({x ? D(x) : nullptr, y ? D(y) : nullptr, D(z), a, b, (uint8_t)op});
  return true;
}

bool NvQueue::reduce(int op, N_Vector x, N_Vector y, double *value) {
  const _generic_N_Vector_Ops *o = x->ops;
  const bool own = op == R_DOT      ? o->nvdotprod == N_VDotProd_PihmGpu
                   : op == R_WSQ    ? o->nvwrmsnorm == N_VWrmsNorm_PihmGpu
                   : op == R_MAXABS ? o->nvmaxnorm == N_VMaxNorm_PihmGpu
                                    : o->nvmin == N_VMin_PihmGpu;
  // with nothing queued the vector's own kernel is the shorter one
  if (!own || (empty() && !failed) || !take(x, y, nullptr)) return false;
  if (q.nred > 0) {  // its value is the first one's
    flush();
  }
  Scratch &s = fam->scratch;
  push_red({D(x), y ? D(y) : nullptr, s.result, 0, op, 0});
  const bool ok = launch(true) == 0;
  *value = ok ? s.host[0] : NAN;
  return true;
}

bool NvQueue::accepts(N_Vector v) const {
  const _generic_N_Vector_Ops *o = v->ops;
  return o->nvgetvectorid == N_VGetVectorID_PihmGpu && o->nvwrmsnorm == N_VWrmsNorm_PihmGpu &&
         o->nvdotprod == N_VDotProd_PihmGpu && o->nvmin == N_VMin_PihmGpu && o->nvprod == N_VProd_PihmGpu && L(v) > 0;
}

bool NvQueue::min_wsq(N_Vector m, N_Vector x, N_Vector w, double *mn, double *sum, const unsigned int *dev_word,
                      unsigned int *word_out) {
  if (!take(x, w, m)) return false;
  if (q.nred > 0) flush();
  Scratch &s = fam->scratch;
  if (m) push_red({D(m), nullptr, s.result, 0, R_MIN, 0});
  push_red({D(x), D(w), s.result, 0, R_WSQ, 0});
  const bool ok = launch(true, -1, dev_word) == 0;
  if (m) *mn = ok ? s.host[0] : NAN;
  *sum = ok ? s.host[m ? 1 : 0] : NAN;
  if (dev_word) *word_out = ok ? *(const unsigned int *)(s.host + 2 + PIHM_NV_SLOTS) : ~0u;
  return true;
}

bool NvQueue::reduce_slot(int op, N_Vector x, N_Vector y, int slot) {
  if (slot < 0 || slot >= PIHM_NV_SLOTS || !take(x, y, nullptr)) return false;
  push_red({D(x), D(y), fam->scratch.slots + 2 * slot, op == R_WSQ ? q.n : 0, op, 0});
  return true;
}

bool NvQueue::fetch(N_Vector v, int count, double *out, const unsigned int *dev_word, unsigned int *word_out,
                    int *rc) {
  if ((q.nred == 0 && !failed) || count < 0 || count > PIHM_NV_SLOTS || !take(v, nullptr, nullptr)) return false;
  Scratch &s = fam->scratch;
  *rc = -2;
  if (launch(true, count, dev_word)) return true;
  for (int i = 0; i < count; i++) out[i] = s.host[2 + i];
  if (dev_word) *word_out = *(const unsigned int *)(s.host + 2 + PIHM_NV_SLOTS);
  *rc = 0;
  return true;
}

}  // namespace pihm_nv
