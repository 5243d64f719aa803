// Device side of the batch engine: the arena that holds many watersheds'
// meshes, CVODE vectors and right-hand-side staging, and the per-round
// "program" that applies each watershed's queued vector operations.
//
// One round executes, for every watershed that is waiting on the device, the
// element-wise N_Vector operations its integrator issued since it last
// suspended, followed by the operation it suspended on: a reduction (WRMS
// norm, dot product, max norm, min) or a right-hand-side evaluation.  The
// program kernel runs all the watersheds' programs in one launch; the
// right-hand side then runs once over the whole arena for the watersheds that
// asked for it.
//
// Each watershed's vectors are contiguous ranges of the vector slots, and the
// program kernel gives watershed s the same number of blocks, the same
// grid-stride element order and the same block and last-block combination as
// the single-vector reduction kernel over a vector of that length.  Together
// with the shared element-wise arithmetic (nv_ops.cuh) and the shared
// right-hand-side kernels, a watershed's trajectory in a batch is bit-for-bit
// the one the single-watershed library computes for it, whatever else shares
// the batch.
#pragma once

#include <cstdint>

#include "nv_select.h"
#include "pihm_internal.h"

namespace pihm {
namespace batch {

constexpr int kVecSlots = 24;    // CVODE vectors per watershed (21 used)
constexpr int kMaxProgOps = 48;  // element-wise operations queued per round and watershed

// Operation codes below 32 are the element-wise N_Vector operations (EwOp).
enum : uint8_t {
  OP_STAGE_IN = 32,  // rhs_in[global position of entry j] = x[j]
  OP_STAGE_OUT,      // z[j] = rhs_out[global position of entry j]
  OP_FORCING,        // element j: pcpdrp = a, edir = b, ett = c
  OP_WS0,            // element j: ws0_surf = x[j]    (post-step update)
  OP_RECORD          // rec[i0] = rivflow[DOWN_CHANL2CHANL][segment i1]
};

struct Op {
  uint8_t code, x, y, z;  // vector slots
  int32_t i0, i1, pad;
  double a, b, c;
};

// A watershed's place in the arena.
struct SysInfo {
  int64_t off;                   // first entry of its vectors in every slot
  int32_t neq, ne, nr, eoff, roff;
  int32_t nblk;                  // blocks of its reductions (red_grid_for(neq))
  int64_t rec_off;               // first entry of its hydrograph record
};

// Two reductions in one: the minimum of rx, and the sum of squares of ry * rw.
constexpr int kRedMinWsq = 32;

// One watershed's work in one round.
struct RoundSys {
  int32_t sys, prog_off, prog_len;
  int32_t red;      // -1: none, else a pihm_nv::RedOp (R_DOT, R_MAXABS, R_WSQ, R_MIN) or kRedMinWsq
  int32_t bstart;   // first block of the program kernel that works on it
  uint8_t rx, ry, rw, pad;
};

struct DeviceArena {
  DevMesh m;            // capacities in ne, nr, nedge, nbank; launch extents = high-water marks
  double *vec;          // [kVecSlots][neq_cap]
  int64_t neq_cap;
  double *rhs_in, *rhs_out;  // [3 ne_cap + 2 nr_cap], the single-watershed state layout
  SysInfo *sysinfo;     // [max_sys]
  double *partials;     // [max_sys][2 * kMaxBlocks]
  unsigned int *tickets;  // [max_sys]
  double *results;      // [max_sys][2], pinned host memory
  unsigned int *done;   // watersheds of the round whose reduction is finished
  double *rec;          // hydrograph records
  RoundSys *round;      // round list, then the ops, one upload per round
  Op *ops;
  int max_sys;
};

// A round's upload from pinned host memory by a kernel that the program
// kernel can start beside (two copies before it and one behind it, with a
// synchronisation, cost about 10 us of a round's 47): n1 bytes at offset 0 and n2 at
// offset off2 of both, multiples of 16; zero words are cleared.
cudaError_t launch_upload(const char *host, char *dev, size_t n1, size_t off2, size_t n2, unsigned int *zero, int nzero,
                          cudaStream_t st);

// Run one round's programs: nrs watersheds over nblocks blocks in total.
// variant 0, 1, 2: entries a thread keeps in flight (1, 2, 4); same results.
// flag: with every watershed of the round ending in a reduction, the last of
// them hands seq to the host (host_flag.h); null: launch_round_done does.
constexpr int kProgramVariants = 3;
// A fourth layout, same results: one warp of the reduction order a block, its
// threads' four entries on four warps.  A warp has one FP64 instruction in
// flight (69 clocks) and an SM takes one every 20, so a round that leaves the
// SMs short of warps is bound by that latency: model steps of 8 watersheds of
// 17,566 elements 7.5 -> 6.2 ms, of 20 of 104,308 (rounds of up to 315
// blocks) 11.4 -> 10.5 ms.  From about 400 blocks the FP64 pipe is full either
// way (24 of 187,100: 12.1 ms with rounds up to 400 blocks spread, 12.5 with
// all or none).  Its partial values need a watershed of kMaxBlocks / 8 blocks
// or fewer.
constexpr int kProgramSpread = 3;
constexpr int kSpreadBlocks = 400;
cudaError_t launch_program(const DeviceArena &a, int nrs, int nblocks, int variant, uint64_t *flag, uint64_t seq,
                           cudaStream_t st);

// Behind a round's last kernel: n words to the host, then seq.
cudaError_t launch_round_done(const unsigned int *words, unsigned int *host, int n, uint64_t *flag, uint64_t seq,
                              cudaStream_t st);

// One part of a watershed's upload: bytes from src (host memory) to dst
// (arena), 32-bit indices moved to the watershed's ranges on the way.
enum UploadOp : int32_t {
  UP_COPY = 0,
  UP_FILL,   // a, n times; src unused
  UP_ADD,    // v + a
  UP_SLOT,   // -1 stays, else v + a
  UP_DOWN,   // v > 0: v + a, else v
  UP_NABR,   // v >= 0: v + a; the boundary stays; a river segment moves by b
  UP_EDGE    // a signed one-based edge: v > 0: v + a, v < 0: v - a
};
struct CopyDesc {
  const void *src;
  void *dst;
  uint64_t bytes;
  int32_t op, a, b, pad;
};
PIHM_HD inline int32_t upload_index(int op, int32_t v, int32_t a, int32_t b) {
  switch (op) {
    case UP_FILL: return a;
    case UP_ADD: return v + a;
    case UP_SLOT: return v < 0 ? v : v + a;
    case UP_DOWN: return v > 0 ? v + a : v;
    case UP_NABR: return v >= 0 ? v + a : (v == kBoundary ? v : v - b);
    default: return v > 0 ? v + a : (v < 0 ? v - a : 0);
  }
}
// Takes every descriptor with one kernel that reads the host memory
// directly.  Only for a device that can access pageable host memory
// (cudaDevAttrPageableMemoryAccess): desc and every src may be ordinary
// host allocations, and they must stay valid until the stream has passed
// the kernel.
cudaError_t launch_gather_host(const CopyDesc *desc, int n, uint64_t max_bytes, cudaStream_t st);

}  // namespace batch


}  // namespace pihm
