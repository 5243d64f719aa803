// The batch engine's program kernel (batch_device.h).
#include "batch_device.h"
#include "host_flag.h"
#include "nv_ops.cuh"

namespace pihm {
namespace batch {

using namespace pihm_nv;

namespace {

// Position of entry j of a watershed's state vector in the arena-wide
// right-hand-side staging vector, which has the single-watershed layout
// [surf | unsat | gw] over ne_cap elements and [stage | rivgw] over nr_cap
// segments.
__device__ __forceinline__ long long stage_pos(const SysInfo &s, long long j, long long ne_cap,
                                               long long nr_cap) {
  const long long ne = s.ne;
  if (j < 3 * ne) {
    const long long p = (j >= ne) + (j >= 2 * ne);
    return p * ne_cap + s.eoff + (j - p * ne);
  }
  const long long jr = j - 3 * ne;
  const long long q = (jr >= s.nr);
  return 3 * ne_cap + q * nr_cap + s.roff + (jr - q * s.nr);
}

// A thread works on kU grid-stride iterations together, so that the loads of
// kU entries are in flight at once; the reduction still accumulates them in
// grid-stride order, so every kU gives the same bits.  The batch engine's
// tuner picks kU (1, 2 or 4) by timing.

// z = OP(a, b, x, y, z) for a run-time operation code
__device__ __forceinline__ double ew_eval_rt(int op, double a, double b, double x, double y, double z) {
  switch (op) {
    case EW_LIN: return ew_eval<EW_LIN>(a, b, x, y, z);
    case EW_LIN1: return ew_eval<EW_LIN1>(a, b, x, y, z);
    case EW_LIN2: return ew_eval<EW_LIN2>(a, b, x, y, z);
    case EW_SUM: return ew_eval<EW_SUM>(a, b, x, y, z);
    case EW_DIFF: return ew_eval<EW_DIFF>(a, b, x, y, z);
    case EW_SCALESUM: return ew_eval<EW_SCALESUM>(a, b, x, y, z);
    case EW_SCALEDIFF: return ew_eval<EW_SCALEDIFF>(a, b, x, y, z);
    case EW_AXPY: return ew_eval<EW_AXPY>(a, b, x, y, z);
    case EW_AXPY1: return ew_eval<EW_AXPY1>(a, b, x, y, z);
    case EW_AXPYM1: return ew_eval<EW_AXPYM1>(a, b, x, y, z);
    case EW_CONST: return ew_eval<EW_CONST>(a, b, x, y, z);
    case EW_PROD: return ew_eval<EW_PROD>(a, b, x, y, z);
    case EW_DIV: return ew_eval<EW_DIV>(a, b, x, y, z);
    case EW_SCALE: return ew_eval<EW_SCALE>(a, b, x, y, z);
    case EW_COPY: return ew_eval<EW_COPY>(a, b, x, y, z);
    case EW_NEG: return ew_eval<EW_NEG>(a, b, x, y, z);
    case EW_ABS: return ew_eval<EW_ABS>(a, b, x, y, z);
    case EW_INV: return ew_eval<EW_INV>(a, b, x, y, z);
    case EW_ADDCONST: return ew_eval<EW_ADDCONST>(a, b, x, y, z);
    default: return ew_eval<EW_COMPARE>(a, b, x, y, z);
  }
}

// Apply one operation to the entries j[0..nu).  base points at the
// watershed's entry 0 in vector slot 0; slots are vs entries apart.
template <int kU>
__device__ __forceinline__ void exec_op(const Op &o, const DeviceArena &A, const SysInfo &S, double *base,
                                        long long vs, const long long (&j)[kU], int nu) {
  if (o.code < EW_COUNT) {
    const bool rx = ew_reads_x(o.code), ry = ew_reads_y(o.code), rz = ew_reads_z(o.code);
    const double *x = base + o.x * vs, *y = base + o.y * vs;
    double *z = base + o.z * vs;
    double xv[kU], yv[kU], zv[kU];
#pragma unroll
    for (int u = 0; u < kU; u++) {
      xv[u] = (u < nu && rx) ? x[j[u]] : 0.0;
      yv[u] = (u < nu && ry) ? y[j[u]] : 0.0;
      zv[u] = (u < nu && rz) ? z[j[u]] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kU; u++)
      if (u < nu) z[j[u]] = ew_eval_rt(o.code, o.a, o.b, xv[u], yv[u], zv[u]);
    return;
  }
  switch (o.code) {
    case OP_STAGE_IN: {
      double v[kU];
#pragma unroll
      for (int u = 0; u < kU; u++)
        if (u < nu) v[u] = base[o.x * vs + j[u]];
#pragma unroll
      for (int u = 0; u < kU; u++)
        if (u < nu) A.rhs_in[stage_pos(S, j[u], A.m.ne, A.m.nr)] = v[u];
      break;
    }
    case OP_STAGE_OUT: {
      double v[kU];
#pragma unroll
      for (int u = 0; u < kU; u++)
        if (u < nu) v[u] = A.rhs_out[stage_pos(S, j[u], A.m.ne, A.m.nr)];
#pragma unroll
      for (int u = 0; u < kU; u++)
        if (u < nu) base[o.z * vs + j[u]] = v[u];
      break;
    }
    case OP_FORCING:
#pragma unroll
      for (int u = 0; u < kU; u++)
        if (u < nu && j[u] < S.ne) {
          const long long g = S.eoff + j[u];
          ((double *)A.m.pcpdrp)[g] = o.a;
          ((double *)A.m.edir)[g] = o.b;
          ((double *)A.m.ett)[g] = o.c;
        }
      break;
    case OP_WS0:
#pragma unroll
      for (int u = 0; u < kU; u++)
        if (u < nu && j[u] < S.ne) ((double *)A.m.ws0_surf)[S.eoff + j[u]] = base[o.x * vs + j[u]];
      break;
    case OP_RECORD:
      if (j[0] == 0) A.rec[S.rec_off + o.i0] = A.m.rivflow[(long long)DOWN_CHANL2CHANL * A.m.nr + S.roff + o.i1];
      break;
    default: break;
  }
}

// kU 0: spread over 128-thread blocks (run_warp)
constexpr int kSpreadThreads = 128;

// One block of one watershed's program: the element-wise operations over the
// block's grid-strided entries, then (RED >= 0) the reduction, combined
// exactly as the single-vector reduction kernel combines it.
template <int RED>
__device__ __forceinline__ Pair last_block(const double *partials, int nblk, Pair *sh) {
  Pair v = red_identity<RED>();
  for (int q = threadIdx.x; q < nblk; q += blockDim.x)
    v = red_combine<RED>(v, Pair{((const volatile double *)partials)[q], 0.0});
  return red_block<RED>(v, sh);
}

// A watershed's result is with the host: the last one of the round says so.
__device__ __forceinline__ void round_end(const DeviceArena &A, int nrs, uint64_t *flag, uint64_t seq) {
  if (!flag) return;
  __threadfence_system();
  if (atomicAdd(A.done, 1u) == (unsigned)nrs - 1) {
    *A.done = 0u;
    __threadfence_system();
    pihm::host_flag_set(flag, seq);
  }
}

// A block's shared memory, one for every reduction it may run: a round's
// watersheds are bounded by what it and the programs leave of 48 KB.
struct BlockShared {
  Pair a[kThreads / 32], b[kThreads / 32];
  bool last;
};

// RED2 >= 0: a second reduction, of A.vec slots ry and rw.
template <int kU, int RED, int RED2 = -1>
__device__ void run_block(const DeviceArena &A, const RoundSys &R, const SysInfo &S, const Op *prog, int b, int nrs,
                          uint64_t *flag, uint64_t seq, BlockShared &bs) {
  Pair *const sh = bs.a, *const sh2 = bs.b;
  bool &last = bs.last;
  const long long vs = A.neq_cap;
  double *base = A.vec + S.off;
  const int nops = R.prog_len;
  const long long n = S.neq;
  const long long stride = (long long)S.nblk * kThreads;
  constexpr int R2 = RED2 >= 0 ? RED2 : 0;
  Pair acc = red_identity<(RED >= 0 ? RED : 0)>(), acc2 = red_identity<R2>();
  for (long long j0 = (long long)b * kThreads + threadIdx.x; j0 < n; j0 += kU * stride) {
    long long j[kU];
    int nu = 0;
#pragma unroll
    for (int u = 0; u < kU; u++) {
      j[u] = j0 + u * stride;
      nu += (j[u] < n);
    }
    for (int p = 0; p < nops; p++) exec_op<kU>(prog[p], A, S, base, vs, j, nu);
    if (RED >= 0) {
      double xv[kU], yv[kU];
#pragma unroll
      for (int u = 0; u < kU; u++)
        if (u < nu) {
          xv[u] = base[R.rx * vs + j[u]];
          yv[u] = (RED == R_DOT || RED == R_WSQ) ? base[R.ry * vs + j[u]] : 0.0;
        }
#pragma unroll
      for (int u = 0; u < kU; u++)
        if (u < nu) acc = red_combine<RED>(acc, red_term<RED>(xv[u], yv[u]));
    }
    if (RED2 >= 0) {
      double xv[kU], yv[kU];
#pragma unroll
      for (int u = 0; u < kU; u++)
        if (u < nu) {
          xv[u] = base[R.ry * vs + j[u]];
          yv[u] = base[R.rw * vs + j[u]];
        }
#pragma unroll
      for (int u = 0; u < kU; u++)
        if (u < nu) acc2 = red_combine<R2>(acc2, red_term<R2>(xv[u], yv[u]));
    }
  }
  if (RED < 0) return;
  acc = red_block<RED>(acc, sh);
  if (RED2 >= 0) acc2 = red_block<R2>(acc2, sh2);
  double *partials = A.partials + (long long)R.sys * 2 * kMaxBlocks;
  unsigned int *ticket = A.tickets + R.sys;
  if (threadIdx.x == 0) {
    partials[b] = acc.v;
    if (RED2 >= 0) partials[kMaxBlocks + b] = acc2.v;
    __threadfence();
    const unsigned int t = atomicAdd(ticket, 1u);
    last = (t == (unsigned)S.nblk - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  const Pair v = last_block<RED>(partials, S.nblk, sh);
  Pair v2 = {0.0, 0.0};
  if (RED2 >= 0) v2 = last_block<R2>(partials + kMaxBlocks, S.nblk, sh2);
  if (threadIdx.x == 0) {
    A.results[2 * R.sys] = v.v;
    A.results[2 * R.sys + 1] = v2.v;
    *ticket = 0u;
    round_end(A, nrs, flag, seq);
  }
}

// The same for a block of 128 threads that carries one warp of the reduction
// order: the four entries a thread of that order accumulates go to four warps
// (nvector.cu, k_seq).  One pass: at most kMaxBlocks / 8 blocks a watershed.
template <int RED, int RED2 = -1>
__device__ void run_warp(const DeviceArena &A, const RoundSys &R, const SysInfo &S, const Op *prog, int vw, int nrs,
                         uint64_t *flag, uint64_t seq) {
  constexpr int R0 = RED >= 0 ? RED : 0, R1 = RED2 >= 0 ? RED2 : 0, NR = RED < 0 ? 0 : (RED2 < 0 ? 1 : 2);
  __shared__ double term[2][kSpreadThreads];
  __shared__ double sh[2][8];
  __shared__ bool last;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const long long vs = A.neq_cap, n = S.neq, stride = (long long)S.nblk * kThreads;
  double *base = A.vec + S.off;
  const long long j0 = (long long)vw * 32 + lane;
  const long long j[1] = {j0 + wid * stride};
  if (j[0] < n) {
    for (int p = 0; p < R.prog_len; p++) exec_op<1>(prog[p], A, S, base, vs, j, 1);
    if (NR > 0) {
      const double x = base[R.rx * vs + j[0]];
      const double y = (R0 == R_DOT || R0 == R_WSQ) ? base[R.ry * vs + j[0]] : 0.0;
      term[0][tid] = red_term<R0>(x, y).v;
      if (NR > 1) term[1][tid] = red_term<R1>(base[R.ry * vs + j[0]], base[R.rw * vs + j[0]]).v;
    }
  }
  if (NR == 0) return;
  double *part = A.partials + (long long)R.sys * 2 * kMaxBlocks;
  __syncthreads();
  if (wid < NR) {
    Pair acc = wid == 0 ? red_identity<R0>() : red_identity<R1>();
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (j0 + u * stride < n) {
        const Pair t = {term[NR > 1 ? wid : 0][u * 32 + lane], 0.0};
        if (u == 0) acc = wid == 0 ? red_first<R0>(t) : red_first<R1>(t);
        else acc = wid == 0 ? red_combine<R0>(acc, t) : red_combine<R1>(acc, t);
      }
    const double v = wid == 0 ? warp_tree<R0>(acc.v) : warp_tree<R1>(acc.v);
    if (lane == 0) part[wid * kMaxBlocks + vw] = v;
  }
  __threadfence();
  __syncthreads();
  unsigned int *ticket = A.tickets + R.sys;
  if (tid == 0) last = atomicAdd(ticket, 1u) == (unsigned)S.nblk * 8 - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  tree_last<R0, true, kSpreadThreads>(S.nblk, part, sh[0]);
  if (NR > 1) tree_last<R1, true, kSpreadThreads>(S.nblk, part + kMaxBlocks, sh[1]);
  __syncthreads();
  if (tid == 0) {
    A.results[2 * R.sys] = eight_tree<R0>(sh[0]);
    A.results[2 * R.sys + 1] = NR > 1 ? eight_tree<R1>(sh[1]) : 0.0;
    *ticket = 0u;
    round_end(A, nrs, flag, seq);
  }
}

template <int kU>
__global__ void __launch_bounds__(kU == 0 ? kSpreadThreads : kThreads, (kU == 0 ? 8 : (kU == 1 ? 6 : (kU == 2 ? 5 : 3)))) k_program(DeviceArena A, int nrs,
                                                                                             uint64_t *flag,
                                                                                             uint64_t seq) {
  // launched beside the upload it reads (launch_program)
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // Stage the round's block ranges and then this block's program in shared
  // memory: one coalesced pass each instead of a chain of dependent global
  // loads before any entry is touched.
  extern __shared__ __align__(16) unsigned char smem[];
  Op *s_ops = reinterpret_cast<Op *>(smem);
  int32_t *s_bstart = reinterpret_cast<int32_t *>(smem + sizeof(Op) * kMaxProgOps);
  for (int i = threadIdx.x; i < nrs; i += blockDim.x) s_bstart[i] = A.round[i].bstart;
  __syncthreads();
  int lo = 0, hi = nrs - 1;
  const int blk = kU == 0 ? blockIdx.x / 8 : blockIdx.x;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (s_bstart[mid] <= blk) lo = mid;
    else hi = mid - 1;
  }
  const RoundSys R = A.round[lo];
  const SysInfo S = A.sysinfo[R.sys];
  const int b = blk - R.bstart;
  if (b >= S.nblk) return;
  {
    const double *src = reinterpret_cast<const double *>(A.ops + R.prog_off);
    double *dst = reinterpret_cast<double *>(s_ops);
    const int nw = R.prog_len * (int)(sizeof(Op) / sizeof(double));
    for (int i = threadIdx.x; i < nw; i += blockDim.x) dst[i] = src[i];
  }
  __syncthreads();
  if constexpr (kU == 0) {
    const int vw = b * 8 + blockIdx.x % 8;
    switch (R.red) {
      case R_DOT: run_warp<R_DOT>(A, R, S, s_ops, vw, nrs, flag, seq); break;
      case R_MAXABS: run_warp<R_MAXABS>(A, R, S, s_ops, vw, nrs, flag, seq); break;
      case R_WSQ: run_warp<R_WSQ>(A, R, S, s_ops, vw, nrs, flag, seq); break;
      case R_MIN: run_warp<R_MIN>(A, R, S, s_ops, vw, nrs, flag, seq); break;
      case kRedMinWsq: run_warp<R_MIN, R_WSQ>(A, R, S, s_ops, vw, nrs, flag, seq); break;
      default: run_warp<-1>(A, R, S, s_ops, vw, nrs, flag, seq); break;
    }
  } else {
    __shared__ BlockShared bs;
    switch (R.red) {
      case R_DOT: run_block<kU, R_DOT>(A, R, S, s_ops, b, nrs, flag, seq, bs); break;
      case R_MAXABS: run_block<kU, R_MAXABS>(A, R, S, s_ops, b, nrs, flag, seq, bs); break;
      case R_WSQ: run_block<kU, R_WSQ>(A, R, S, s_ops, b, nrs, flag, seq, bs); break;
      case R_MIN: run_block<kU, R_MIN>(A, R, S, s_ops, b, nrs, flag, seq, bs); break;
      case kRedMinWsq: run_block<kU, R_MIN, R_WSQ>(A, R, S, s_ops, b, nrs, flag, seq, bs); break;
      default: run_block<kU, -1>(A, R, S, s_ops, b, nrs, flag, seq, bs); break;
    }
  }
}

}  // namespace

static_assert(sizeof(Op) == 40 && sizeof(Op) % sizeof(double) == 0, "Op is staged as doubles");

// blockIdx.y picks the descriptor, blockIdx.x a kGatherChunk-byte chunk of
// it; indices word by word, else 8-byte words where source, destination and size allow, else 4-byte
// words, else bytes
constexpr uint64_t kGatherChunk = 64 * 1024;

__global__ void __launch_bounds__(256) k_gather_host(const CopyDesc *desc, int n) {
  const CopyDesc d = desc[blockIdx.y];
  const uint64_t lo = (uint64_t)blockIdx.x * kGatherChunk;
  if (lo >= d.bytes) return;
  const uint64_t hi = min(d.bytes, lo + kGatherChunk);
  const uintptr_t align = (uintptr_t)d.src | (uintptr_t)d.dst | (uintptr_t)d.bytes;
  const char *src = (const char *)d.src;
  char *dst = (char *)d.dst;
  if (d.op != UP_COPY) {  // 32-bit words
    for (uint64_t b = lo + 4 * (uint64_t)threadIdx.x; b < hi; b += 4 * (uint64_t)blockDim.x)
      *(int32_t *)(dst + b) = upload_index(d.op, d.op == UP_FILL ? 0 : *(const int32_t *)(src + b), d.a, d.b);
    return;
  }
  if ((align & 7) == 0) {
    for (uint64_t b = lo + 8 * (uint64_t)threadIdx.x; b < hi; b += 8 * (uint64_t)blockDim.x)
      *(uint64_t *)(dst + b) = *(const uint64_t *)(src + b);
  } else if ((align & 3) == 0) {
    for (uint64_t b = lo + 4 * (uint64_t)threadIdx.x; b < hi; b += 4 * (uint64_t)blockDim.x)
      *(uint32_t *)(dst + b) = *(const uint32_t *)(src + b);
  } else {
    for (uint64_t b = lo + threadIdx.x; b < hi; b += blockDim.x) dst[b] = src[b];
  }
}

cudaError_t launch_gather_host(const CopyDesc *desc, int n, uint64_t max_bytes, cudaStream_t st) {
  if (n <= 0 || max_bytes == 0) return cudaSuccess;
  if (n > 65535) return cudaErrorInvalidValue;
  const dim3 grid((unsigned)((max_bytes + kGatherChunk - 1) / kGatherChunk), (unsigned)n);
  k_gather_host<<<grid, 256, 0, st>>>(desc, n);
  return cudaGetLastError();
}

__global__ void __launch_bounds__(256) k_upload(const int4 *host, int4 *dev, int n1, int off2, int n2,
                                                unsigned int *zero, int nzero) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int i0 = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  for (int i = i0; i < n1 + n2; i += step) {
    const int k = i < n1 ? i : off2 + (i - n1);
    dev[k] = host[k];
  }
  for (int i = i0; i < nzero; i += step) zero[i] = 0u;
}

cudaError_t launch_upload(const char *host, char *dev, size_t n1, size_t off2, size_t n2, unsigned int *zero, int nzero,
                          cudaStream_t st) {
  const int words = (int)((n1 + n2) / 16);
  const int grid = words < 256 * 32 ? (words + 255) / 256 : 32;
  k_upload<<<grid, 256, 0, st>>>((const int4 *)host, (int4 *)dev, (int)(n1 / 16), (int)(off2 / 16), (int)(n2 / 16),
                                 zero, nzero);
  return cudaGetLastError();
}

__global__ void __launch_bounds__(256) k_round_done(const unsigned int *words, unsigned int *host, int n, uint64_t *flag,
                                                    uint64_t seq) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) host[i] = words[i];
  __threadfence_system();
  __syncthreads();
  if (threadIdx.x == 0) pihm::host_flag_set(flag, seq);
}

cudaError_t launch_round_done(const unsigned int *words, unsigned int *host, int n, uint64_t *flag, uint64_t seq,
                              cudaStream_t st) {
  k_round_done<<<1, 256, 0, st>>>(words, host, n, flag, seq);
  return cudaGetLastError();
}

cudaError_t launch_program(const DeviceArena &a, int nrs, int nblocks, int variant, uint64_t *flag, uint64_t seq,
                           cudaStream_t st) {
  if (nrs <= 0 || nblocks <= 0) return cudaSuccess;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)nblocks);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = sizeof(Op) * kMaxProgOps + sizeof(int32_t) * (size_t)nrs;
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  if (variant == kProgramSpread) {
    cfg.gridDim = dim3((unsigned)nblocks * (kThreads / 32));
    cfg.blockDim = dim3(kSpreadThreads);
    return launched(cudaLaunchKernelEx(&cfg, k_program<0>, a, nrs, flag, seq));
  }
  if (variant == 0) return launched(cudaLaunchKernelEx(&cfg, k_program<1>, a, nrs, flag, seq));
  if (variant == 1) return launched(cudaLaunchKernelEx(&cfg, k_program<2>, a, nrs, flag, seq));
  return launched(cudaLaunchKernelEx(&cfg, k_program<4>, a, nrs, flag, seq));
}

}  // namespace batch
}  // namespace pihm
