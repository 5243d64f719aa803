// Warp-shuffle / block reduction helpers shared by the N_Vector kernels.
#pragma once

#include <cmath>

#include "nv_select.h"

namespace pihm_nv {

struct Pair {
  double v;
  double f;  // flag channel (found / failed)
};

template <int OP>
__device__ __forceinline__ Pair red_identity() {
  if (OP == R_MAXABS) return {0.0, 0.0};
  if (OP == R_MIN || OP == R_MINQ) return {INFINITY, 0.0};
  return {0.0, 0.0};
}

template <int OP>
__device__ __forceinline__ Pair red_combine(Pair p, Pair q) {
  if (OP == R_MAXABS) {
    // fmax of values that are not negative (a NaN loses, as in fmax), by
    // their bit patterns
    const unsigned long long a = (unsigned long long)__double_as_longlong(p.v);
    const unsigned long long b = (unsigned long long)__double_as_longlong(q.v);
    const unsigned long long inf = 0x7FF0000000000000ull;
    return {__longlong_as_double((long long)((a > inf || (b <= inf && b > a)) ? b : a)), 0.0};
  }
  if (OP == R_MIN || OP == R_MINQ) return {fmin(p.v, q.v), fmax(p.f, q.f)};
  if (OP == R_INVTEST || OP == R_CONSTR) return {0.0, fmax(p.f, q.f)};
  return {__dadd_rn(p.v, q.v), 0.0};
}

template <int OP>
__device__ __forceinline__ Pair red_block(Pair v, Pair *sh) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    Pair q;
    q.v = __shfl_down_sync(0xffffffffu, v.v, o);
    q.f = __shfl_down_sync(0xffffffffu, v.f, o);
    v = red_combine<OP>(v, q);
  }
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  if (wid == 0) {
    v = (lane < (int)(blockDim.x >> 5)) ? sh[lane] : red_identity<OP>();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      Pair q;
      q.v = __shfl_down_sync(0xffffffffu, v.v, o);
      q.f = __shfl_down_sync(0xffffffffu, v.f, o);
      v = red_combine<OP>(v, q);
    }
  }
  return v;
}

// p combined with the identity, as the first step of a sum or of a tree over
// fewer values than lanes: of the sums only -0 changes.
template <int RED>
__device__ __forceinline__ Pair red_first(Pair p) {
  if (RED == R_DOT || RED == R_WSQ) {
    const long long b = __double_as_longlong(p.v);
    return {__longlong_as_double(b == (long long)0x8000000000000000ull ? 0 : b), 0.0};
  }
  return red_combine<RED>(red_identity<RED>(), p);
}

// The shuffle tree of one warp, and the tree over a block's eight warp
// values, as red_block makes them.
template <int RED>
__device__ __forceinline__ double warp_tree(double x) {
  Pair v = {x, 0.0};
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const Pair q = {__shfl_down_sync(0xffffffffu, v.v, o), 0.0};
    v = red_combine<RED>(v, q);
  }
  return v.v;
}
template <int RED>
__device__ __forceinline__ double eight_tree(const volatile double *w) {
  Pair v[8];
#pragma unroll
  for (int k = 0; k < 8; k++) v[k] = red_first<RED>({w[k], 0.0});
#pragma unroll
  for (int o = 4; o > 0; o >>= 1)
#pragma unroll
    for (int k = 0; k < o; k++) v[k] = red_combine<RED>(v[k], v[k + o]);
  return v[0].v;
}

// The last block's combination of the partial values of nblk blocks of the
// reduction order, by kT threads; sh holds the eight warps' values then.
// kSpread: `part` has a value per warp of that order, eight a block.
template <int RED, bool kSpread, int kT>
__device__ __forceinline__ void tree_last(int nblk, const double *part, double *sh) {
  const int lane = threadIdx.x & 31;
  for (int vw = threadIdx.x >> 5; vw < 8; vw += kT / 32) {
    double v = red_identity<RED>().v;
    if (vw * 32 < nblk) {
      for (int b = vw * 32 + lane, k = 0; b < nblk; b += kThreads, k++) {
        const Pair t = {kSpread ? eight_tree<RED>(part + 8 * b) : ((const volatile double *)part)[b], 0.0};
        v = k == 0 ? red_first<RED>(t).v : red_combine<RED>({v, 0.0}, t).v;
      }
      v = warp_tree<RED>(v);
    }
    if (lane == 0) sh[vw] = v;
  }
}

}  // namespace pihm_nv
