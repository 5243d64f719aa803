// FP64 right-hand-side kernels of the PIHM hydrologic model for sm_103a.
//
// One evaluation of f(t, y) (the reference ODE(), src/ode.c:4-399) runs as
// one cooperative launch (k_rhs_fused: small meshes) or five programmatic
// dependent launches, with no host synchronisation.  An SM takes an FP64 warp
// instruction every 20 clocks, so the FP64 pipe is the scarce one: the element rows' powers, divisions and
// square roots run in fixed point on the integer pipe (int_math.cuh; the
// divisions and roots IEEE-exact), comparisons and sign flips on the
// integer pipe too (fp64_cmp.h), divisions by static quantities are
// multiplications by reciprocals computed at load, sub-expressions the
// reference re-evaluates (EffKh per edge side, KrFunc/Psi in Infil and
// Recharge) are computed once, and each block ranks its elements by branch
// class so that a warp's lanes share their branches.
//
//   k_elem_prep   per element: clamp y (src/ode.c:25-49), SurfH
//                 (src/hydrol.c:100-134), surface head zmax + surfh and the
//                 macropore-weighted conductivity EffKh(gw)
//                 (src/lat_flow.c:248-277), each computed once per element
//                 instead of once per edge side as in the reference.
//   k_elem_grad   per element: FrictSlope/DhByDl water-surface gradient
//                 (src/lat_flow.c:130-185,239-246) reduced to its magnitude,
//                 with the purely geometric denominators precomputed.
//   k_elem_main   per element: edge fluxes (SubFlowElemToElem,
//                 OvlFlowElemToElem, BoundFluxElem, src/lat_flow.c:285-382),
//                 EtExtract (src/hydrol.c:33-97), Infil/Recharge/EffKinf/AvgKv
//                 (src/vert_flow.c:33-270) and the element rows of ydot
//                 (src/ode.c:111-209) but for the river banks'.
//   k_edge        per interior edge: the Darcy and Manning fluxes, evaluated
//                 once and read with a sign by both elements.
//   k_riv_geom    per segment: channel area and wetted perimeter at the
//                 stage (src/river_flow.c:520-583), once per segment; part
//                 of k_elem_prep's grid.
//   k_river       per segment, in four parts: RiverFlow
//                 (src/river_flow.c:3-94) and RiverToElem (:113-183), ChanLeak,
//                 OutletFlux, BoundFluxRiver; part of k_elem_grad's grid.
//   k_river_rows  per segment: upstream accumulation in reference order
//                 (src/river_flow.c:96-110, a CSR list instead of a serial
//                 loop) and the river rows of ydot (src/ode.c:228-300); part
//                 of k_bank_rows's grid.
//   k_bank_rows   per element with river edges: its rows of ydot from
//                 k_elem_main's sums and the river fluxes.
//
// Infil reads the river-edge overland flux of the previous evaluation
// (src/vert_flow.c:61 runs before src/river_flow.c:159-182 rewrites it); that
// value is the previous evaluation's LEFT/RIGHT_SURF2CHANL in carry_ovl, which
// k_elem_main reads and k_bank_rows then replaces.
#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "fp64_math.cuh"
#include "host_flag.h"
#include "pihm_internal.h"

namespace pihm {

#define RESTRICT __restrict__

// Comparisons go through fp64_cmp.h: the same results as the C operators,
// evaluated on the integer pipe instead of the FP64 pipe.
__device__ __forceinline__ double clamp0(double v) { return cmp::ge0(v) ? v : 0.0; }

// AvgH, src/lat_flow.c:217-237
__device__ __forceinline__ double avg_h_sub(double diff, double hsub, double hnabr) {
  if (cmp::gt0(diff)) return cmp::gt0(hsub) ? hsub : 0.0;
  return cmp::gt0(hnabr) ? hnabr : 0.0;
}

// AvgHsurf, src/lat_flow.c:187-215
__device__ __forceinline__ double avg_h_surf(double diff, double hsurf, double hnabr) {
  if (cmp::gt0(diff)) return cmp::gt_c(hsurf, kDeprStg) ? 1.0 * (hsurf - kDeprStg) : 0.0;
  return cmp::gt_c(hnabr, kDeprStg) ? 1.0 * (hnabr - kDeprStg) : 0.0;
}

// OverLandFlow, src/lat_flow.c:279-283
__device__ __forceinline__ double overland_flow(double avg_h, double grad_h, double avg_sf,
                                                double crossa, double avg_rough) {
  return div_any(crossa * pow_manning(avg_h, kManningSurf) * grad_h, sqrt_any(avg_sf) * avg_rough);
}

// KrFunc (src/soil.c:8-13) and Psi (src/vert_flow.c:272-278) of one
// saturation in [SATMIN, 1], in the reference's own operations:
//   KrFunc = sqrt(satn) (1 - (1 - satn^m)^e) (1 - (1 - satn^m)^e),
//   Psi    = -((1 / satn)^m - 1)^ib / alpha,
// m = beta/(beta - 1), e = (beta - 1)/beta, ib = 1/beta formed at load as
// the reference forms them.  Recharge's head gradient 0.5 deficit + Psi and
// Infil's surfh + zmax - (Psi + zmax - 0.5 dinf) cancel by up to four
// orders of magnitude near equilibrium, so Psi has to carry the reference's
// roundings: each power is correctly rounded but for a rare last bit
// (pow_any), and 1/satn and the division by alpha are IEEE divisions as in
// the reference.  The powers run on the integer pipe.
// sq returns sqrt(satn), which EffKinf's macropore branch needs too.
// satn^m and (1/satn)^m share satn's logarithm: the second is the power of
// the rounded reciprocal fl(1/satn), whose logarithm follows from satn's and
// the exact residual of the division (im::log2k_recip), within the same
// 0.502 ulp as a power of its own.
//
// kr_psi evaluates everything without a branch, so that the root, the
// reciprocal and the two last powers run beside each other, and asks once at
// the end whether an operand was out of a range (a NaN state); kr_psi_slow
// then repeats it operation by operation.
static __device__ __noinline__ void kr_psi_slow(double satn, double vm, double vg_e, double vg_ib, double alpha,
                                                double *satkfunc, double *psi, double *sq) {
  *sq = sqrt_any(satn);
  const double q = div_any(1.0, satn);
  double pm, qm;  // satn^m, (1/satn)^m
  int k, kq;
  int64_t w, wq;
  im::TVal t1, t3;
  if (im::log2k(satn, k, w) && im::mul_t(vm, k, w, t1) && im::log2k_recip(satn, q, k, w, kq, wq) &&
      im::mul_t(vm, kq, wq, t3)) {
    pm = im::exp2k(t1);
    qm = im::exp2k(t3);
  } else {
    pm = pow_any(satn, vm);
    qm = pow_any(q, vm);
  }
  const double t = 1.0 - pow_any(1.0 - pm, vg_e);
  *satkfunc = *sq * t * t;
  *psi = cmp::neg_if(div_any(pow_any(qm - 1.0, vg_ib), alpha), true);
}
__device__ __forceinline__ void kr_psi(double satn, double vm, double vg_e, double vg_ib, double alpha,
                                       double &satkfunc, double &psi, double &sq) {
  int k, kq;
  int64_t w, wq;
  im::TVal t1, t3;
  double q, p1, p3, d;
  bool ok = im::sqrt_i(satn, sq);
  ok &= im::div_i(1.0, satn, q);
  ok &= im::log2k(satn, k, w);
  ok &= im::mul_t(vm, k, w, t1);
  ok &= im::log2k_recip(satn, q, k, w, kq, wq);
  ok &= im::mul_t(vm, kq, wq, t3);
  const double pm = im::exp2k(t1), qm = im::exp2k(t3);  // satn^m, (1/satn)^m
  ok &= im::pow_i(1.0 - pm, vg_e, p1);
  ok &= im::pow_i(qm - 1.0, vg_ib, p3);
  const double t = 1.0 - p1;
  satkfunc = sq * t * t;
  ok &= im::div_i(p3, alpha, d);
  psi = cmp::neg_if(d, true);
  if (!ok) {
    double a, b, c;  // the callers' values stay in registers
    kr_psi_slow(satn, vm, vg_e, vg_ib, alpha, &a, &b, &c);
    satkfunc = a;
    psi = b;
    sq = c;
  }
}

// The evaluation's kernels and the reorderings are programmatic dependent
// launches: each waits for the one before it where it first needs its results,
// the first of an evaluation before anything.  A kernel of the large path lets
// the next one's blocks in once its own are past that wait -- so the kernel two
// ahead is always finished -- and what stands before a wait reads only what an
// earlier evaluation or the caller left.  The last kernel (and k_rhs_fused)
// does not: whatever follows took the places of its own blocks (60,000
// elements, one evaluation after the other: 47 us, 40 without).
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void next_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Batch engine: whether the watershed of item idx sits out this evaluation
// (a free arena slot, or a watershed that did not ask for one).  Always false
// in a single-watershed context.
__device__ __forceinline__ bool skip_item(const DevMesh &m, const int32_t *sys_of, int idx, int *sy) {
  *sy = 0;
  if (!m.active) return false;
  const int s = sys_of[idx];
  *sy = s;
  return s < 0 || !m.active[s];
}

__device__ __forceinline__ void report_err(const DevMesh &m, int sy, unsigned code = kErrNan) {
  atomicOr(m.err_sys ? &m.err_sys[sy] : m.err, code);
}

// Slot of the calling thread in a block's shared-memory work queue when take
// is true (one shared atomic per warp); every thread of the warp calls it.
// Queued work is evaluated densely after a barrier, so a few lanes that need
// an expensive branch do not hold a whole warp on the FP64 pipe.
__device__ __forceinline__ int queue_slot(int *count, bool take) {
  const unsigned lane = threadIdx.x & 31u;
  const unsigned mask = __ballot_sync(0xffffffffu, take);
  int base = 0;
  if (lane == 0 && mask) base = atomicAdd(count, __popc(mask));
  base = __shfl_sync(0xffffffffu, base, 0);
  return base + __popc(mask & ((1u << lane) - 1u));
}

// ---------------------------------------------------------------------------
// k_elem_prep.  Thin surface films (SurfH's square root, about half the
// elements) and water tables inside the macropore zone (EffKh's division,
// about a third) are spread over every warp, so both are queued and
// evaluated densely.
// ---------------------------------------------------------------------------
constexpr int kPrepBlock = 256;
constexpr unsigned kPrepWave = 8 * 152;  // blocks that GB300's SMs hold at once

// SurfH and EffKh of one element (src/hydrol.c:100-134, src/lat_flow.c:248-277):
// what needs no root or division is stored here; thin asks for
// surfh = sqrt(sx), mix for effk = num / den.  EffKh's k1 = kmach*areafv +
// ksath*(1-areafv) and depth - dmac are formed at load (the reference
// evaluates both inline with the same operations).
__device__ __forceinline__ void prep_item(const DevMesh &m, int i, double y_surf, double y_gw, bool &thin, double &sx,
                                          bool &mix, double &num, double &den) {
  const double surfeqv = clamp0(y_surf);
  if (cmp::lt0(surfeqv)) {
    m.surfh[i] = 0.0;
    m.head[i] = 0.0 + m.zmax[i];
  } else if (cmp::le_c(surfeqv, 0.5 * kDeprStg)) {
    thin = true;
    sx = 2.0 * kDeprStg * surfeqv;
  } else {
    const double sh = kDeprStg + (surfeqv - 0.5 * kDeprStg);
    m.surfh[i] = sh;
    m.head[i] = sh + m.zmax[i];
  }
  double gw = clamp0(y_gw);
  gw = cmp::gt0(gw) ? gw : 0.0;
  const double d_dmac = m.d_dmac[i];
  if (cmp::gt_v(gw, d_dmac)) {
    const double d1 = cmp::gt_v(gw, m.depth[i]) ? m.dmac[i] : gw - d_dmac;
    num = m.kh_k1[i] * d1 + m.ksath[i] * d_dmac;
    den = d1 + d_dmac;
    mix = true;
  } else {
    m.effk[i] = m.ksath[i];
  }
}
__device__ __forceinline__ void prep_root(const DevMesh &m, int i, double sx) {
  const double sh = sqrt_any(sx);
  m.surfh[i] = sh;
  m.head[i] = sh + m.zmax[i];
}

// ---------------------------------------------------------------------------
// k_riv_geom: wetted perimeter and cross-section area of every segment at its
// stage (RivPerim / RivCsArea, src/river_flow.c:520-583), once per segment
// and evaluation (k_river needs them for the segment and for its downstream
// neighbour), with the coefficient-only factors formed at load (r_geo*, in
// the order the shape's formula uses them):
//   rectangle  area d c,           perimeter 2 d + c
//   triangle   area d^2 / c,       perimeter 2 d sqrt(1 + c^2) / c
//   quadratic  area 4 d^1.5 / (3 sqrt c),
//              perimeter sqrt(d (1 + 4 c d) / c) + ln(2 sqrt(c d) + sqrt(1 + 4 c d)) / (2 c)
//   cubic      area 3 d^(4/3) / (2 c^(1/3)),
//              perimeter 2 (sqrt(d (1 + 9 c^(2/3) d)) / 3
//                           + ln(3 c^(1/3) sqrt(d) + sqrt(1 + 9 c^(2/3) d)) / (9 c^(1/3)))
// The reference's pow(x, 0.5) is sqrt(x).
// ---------------------------------------------------------------------------
__device__ __forceinline__ double log_of(double x) {
  double sh, lo;
  return log_dd_fast(x, sh, lo) ? sh + lo : log(x);
}

__device__ __forceinline__ void geom_item(const DevMesh &m, const double *y, int s) {
  double d = y[3 * m.ne + s];
  d = cmp::gt0(d) ? d : 0.0;
  const double g0 = m.r_geo0[s];
  double area = 0.0, perim = 0.0;
  switch (m.intrpl_ord[s]) {
    case kRectangle:
      area = d * g0;
      perim = 2.0 * d + g0;
      break;
    case kTriangle:
      area = d * d * g0;
      perim = d * m.r_geo1[s];
      break;
    case kQuadratic:
    case kCubic: {
      // one path for both shapes, so that a warp with segments of both runs
      // the roots and the logarithm once
      const bool cub = m.intrpl_ord[s] == kCubic;
      const double sd = sqrt_any(d), w = 1.0 + m.r_geo1[s] * d;
      const double g2 = m.r_geo2[s], dw = d * w;
      const double root = sqrt_any(cub ? dw : dw * g2);
      const double lg = log_of((cub ? g2 : m.r_geo4[s]) * sd + sqrt_any(w));
      area = cub ? g0 * pow_fast(d, 4.0 / 3.0) : g0 * d * sd;
      perim = cub ? 2.0 * (root * (1.0 / 3.0) + lg * m.r_geo3[s]) : root + lg * m.r_geo3[s];
      break;
    }
  }
  m.r_perim[s] = perim;
  m.r_crossa[s] = area;
}

__global__ void __launch_bounds__(128) k_riv_geom(DevMesh m, const double *RESTRICT y) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  int sy;
  if (s >= m.nr_run || skip_item(m, m.sys_riv, s, &sy)) return;
  geom_item(m, y, s);
}

// ---------------------------------------------------------------------------
// k_river
// ---------------------------------------------------------------------------
struct RivState {
  double stage, gw, zbed, zmin, zmax, length, width, rough;
};

__device__ __forceinline__ RivState load_riv(const DevMesh &m, const double *y, int s) {
  RivState r;
  r.stage = clamp0(y[3 * m.ne + s]);
  r.gw = clamp0(y[3 * m.ne + m.nr + s]);
  r.zbed = m.r_zbed[s];
  r.zmin = m.r_zmin[s];
  r.zmax = m.r_zmax[s];
  r.length = m.r_length[s];
  r.width = m.r_width[s];
  r.rough = m.r_rough[s];
  return r;
}

// OvlFlowElemToRiver, src/river_flow.c:185-255, with the weir coefficient
// cwr 2 sqrt(2 g) length / 3 formed at load (coef)
__device__ __forceinline__ double ovl_elem_to_river(double e_zmax, double e_surfh, const RivState &r,
                                                    double coef) {
  const double zbank = cmp::gt_v(r.zmax, e_zmax) ? r.zmax : e_zmax;
  const double elem_h = e_zmax + e_surfh;
  const double rivseg_h = r.zbed + r.stage;
  // the four cases differ in the head under the root and the head over the
  // bank: one root and one product serve a warp whose lanes take them all
  const bool out = cmp::gt_v(rivseg_h, elem_h);
  if (!out && !cmp::gt_c(e_surfh, kDeprStg)) return 0.0;
  const double high = out ? rivseg_h : elem_h, low = out ? elem_h : rivseg_h;
  const bool drowned = cmp::gt_v(low, zbank);  // the lower side stands above the bank too
  if (!drowned && !cmp::lt_v(zbank, high)) return 0.0;
  const double over = high - zbank;
  const double root = sqrt_any(drowned ? high - low : over);
  return (out ? coef : -coef) * root * over;
}

// ChanFlowElemToRiver, src/river_flow.c:429-460
__device__ __forceinline__ double chan_elem_to_river(double e_gw, double e_zmin, double effk,
                                                     const RivState &r, double r_ksath,
                                                     double inv_distance) {
  const double diff_h = (r.stage + r.zbed) - (e_gw + e_zmin);
  double avg_h;
  if (cmp::gt_v(e_zmin, r.zbed)) avg_h = e_gw;
  else if (cmp::gt_v(e_zmin + e_gw, r.zbed)) avg_h = e_zmin + e_gw - r.zbed;
  else avg_h = 0.0;
  avg_h = avg_h_sub(diff_h, r.stage, avg_h);
  const double grad_h = diff_h * inv_distance;
  const double avg_ksat = 0.5 * (effk + r_ksath);
  return r.length * avg_ksat * grad_h * avg_h;
}

// SubFlowElemToRiver, src/river_flow.c:462-498 (arithmetic mean)
__device__ __forceinline__ double sub_elem_to_river(double e_gw, double e_zmin, double effk,
                                                    const RivState &r, double effk_riv,
                                                    double inv_distance) {
  const double diff_h = (r.gw + r.zmin) - (e_gw + e_zmin);
  double avg_h;
  if (cmp::gt_v(e_zmin, r.zbed)) avg_h = 0.0;
  else if (cmp::gt_v(e_zmin + e_gw, r.zbed)) avg_h = r.zbed - e_zmin;
  else avg_h = e_gw;
  avg_h = avg_h_sub(diff_h, r.gw, avg_h);
  const double avg_ksat = 0.5 * (effk + effk_riv);
  const double grad_h = diff_h * inv_distance;
  return r.length * avg_ksat * grad_h * avg_h;
}

// OutletFlux, src/river_flow.c:333-390
__device__ __forceinline__ void outlet_flux(const DevMesh &m, const RivState &r, int s, int down) {
  const int nr = m.nr;
  double dnf;
  const double depth = m.r_depth[s];
  const double bc = m.river_bc[s];
  if (down == kDirichlet) {
    const double total_h = r.stage + r.zbed;
    const double grad_h = (total_h - bc) * m.r_inv_half_len[s];
    const double avg_perim = m.r_perim[s];
    const double crossa = m.r_crossa[s];
    const double avg_h = cmp::eq0(avg_perim) ? 0.0 : div_any(crossa, avg_perim);
    dnf = overland_flow(avg_h, grad_h, grad_h, crossa, r.rough);
  } else if (down == kNeumann) {
    dnf = -bc;
  } else if (down == kZeroDpthGrad) {
    const double grad_h = (r.zbed - (m.r_node_zmax[s] - depth)) * m.r_inv_half_len[s];
    const double avg_perim = m.r_perim[s];
    const double crossa = m.r_crossa[s];
    dnf = div_any(sqrt_any(grad_h) * crossa *
                      (cmp::gt0(avg_perim) ? pow_manning(div_any(crossa, avg_perim), kManningRiv) : 0.0),
                  r.rough);
  } else {  // kCritDpth (other values are rejected at load)
    const double crossa = m.r_crossa[s];
    dnf = crossa * sqrt_any(kGrav * r.stage);
  }
  m.rivflow[UP_CHANL2CHANL * nr + s] = 0.0;
  m.rivflow[DOWN_CHANL2CHANL * nr + s] = dnf;
}

// A segment's fluxes in four parts that share no result: the channel flux,
// the two banks, and the bed's.  One thread per part: a segment's fluxes are a
// chain of FP64 divisions, roots and a power (18 us for 100 segments or
// 12,000 with one thread per segment), and the parts run beside each other.
// An outlet's channel flux goes with its bed, the shortest part: with the
// channel fluxes of its warp it took the warp 2 us longer than the others.
enum RivPart { PART_CHAN = 0, PART_LEFT, PART_RIGHT, PART_BED, kRivParts };

__device__ __forceinline__ void river_part(const DevMesh &m, const double *y, int s, int part) {
  const int nr = m.nr, ne = m.ne;
  double *F = m.rivflow;
  const RivState r = load_riv(m, y, s);
  if (part == PART_CHAN) {
    const int down = m.down[s];
    if (down <= 0) return;  // an outlet: the bed's part
    double up = 0.0;
    const int bct = m.bctype_riv[s];
    if (bct != 0) {
      // BoundFluxRiver, src/river_flow.c:392-427
      double flux = 0.0;
      const double bc = m.river_bc[s];
      if (bct > 0) {
        const double total_h = r.stage + r.zbed;
        const double grad_h = (total_h - bc) * m.r_inv_half_len[s];
        const double avg_perim = m.r_perim[s];
        const double crossa = m.r_crossa[s];
        const double avg_h = cmp::eq0(avg_perim) ? 0.0 : div_any(crossa, avg_perim);
        flux = overland_flow(avg_h, grad_h, grad_h, crossa, r.rough);
      } else {
        flux = -bc;
      }
      up += flux;
    }
    const int d = down - 1;
    const RivState dn = load_riv(m, y, d);
    const double inv_dist_down = m.r_inv_dist_down[s];
    // ChanFlowRiverToRiver, src/river_flow.c:257-300
    const double total_h = r.stage + r.zbed;
    const double perim = m.r_perim[s];
    const double total_h_down = dn.stage + dn.zbed;
    const double perim_down = m.r_perim[d];
    const double avg_perim = (perim + perim_down) / 2.0;
    const double avg_rough = (r.rough + dn.rough) / 2.0;
    const double diff_h = (m.riv_mode == kKinematic) ? (r.zbed - dn.zbed) : (total_h - total_h_down);
    const double grad_h = diff_h * inv_dist_down;
    const double avg_sf = cmp::gt0(grad_h) ? grad_h : kRivGradMin;
    const double crossa = m.r_crossa[s];
    const double crossa_down = m.r_crossa[d];
    const double avg_crossa = 0.5 * (crossa + crossa_down);
    const double avg_h = cmp::eq0(avg_perim) ? 0.0 : div_any(avg_crossa, avg_perim);
    const double dnf = overland_flow(avg_h, grad_h, avg_sf, crossa, avg_rough);
    F[UP_CHANL2CHANL * nr + s] = up;
    F[DOWN_CHANL2CHANL * nr + s] = dnf;
    return;
  }
  const int L = m.left[s], R = m.right[s];
  const double effk_l = m.effk[L], effk_r = m.effk[R];
  if (part == PART_BED) {
    const int down = m.down[s];
    double aq = 0.0;
    if (down > 0) {
      // SubFlowRiverToRiver, src/river_flow.c:302-331 (arithmetic mean)
      const int d = down - 1;
      const RivState dn = load_riv(m, y, d);
      const double effk = 0.5 * (effk_l + effk_r);
      const double effk_nabr = 0.5 * (m.effk[m.left[d]] + m.effk[m.right[d]]);
      const double total_h = r.gw + r.zmin;
      const double total_h_down = dn.gw + dn.zmin;
      const double avg_wid = (r.width + dn.width) / 2.0;
      const double diff_h = total_h - total_h_down;
      const double avg_h = avg_h_sub(diff_h, r.gw, dn.gw);
      const double grad_h = diff_h * m.r_inv_dist_down[s];
      const double avg_ksat = 0.5 * (effk + effk_nabr);
      aq = avg_ksat * grad_h * avg_h * avg_wid;
    }
    F[DOWN_AQUIF2AQUIF * nr + s] = aq;
    F[UP_AQUIF2AQUIF * nr + s] = 0.0;
    // ChanLeak, src/river_flow.c:500-518
    double diff_h;
    if (cmp::gt0(r.zbed - (r.gw + r.zmin))) diff_h = r.stage;
    else diff_h = r.stage + r.zbed - (r.gw + r.zmin);
    const double grad_h = diff_h * m.r_inv_bedthick[s];
    F[CHANL_LKG * nr + s] = m.r_ksatv[s] * r.width * r.length * grad_h;
    if (down <= 0) outlet_flux(m, r, s, down);
    return;
  }
  // RiverToElem, src/river_flow.c:113-183, one bank
  const bool left = part == PART_LEFT;
  const int e = left ? L : R;
  const double effk_e = left ? effk_l : effk_r;
  const double inv_d = left ? m.r_inv_dist_left[s] : m.r_inv_dist_right[s];
  const double gw_e = clamp0(y[2 * ne + e]), zmin_e = m.zmin[e];
  F[(left ? LEFT_SURF2CHANL : RIGHT_SURF2CHANL) * nr + s] =
      ovl_elem_to_river(m.zmax[e], m.surfh[e], r, m.r_ovl_coef[s]);
  F[(left ? LEFT_AQUIF2CHANL : RIGHT_AQUIF2CHANL) * nr + s] =
      chan_elem_to_river(gw_e, zmin_e, effk_e, r, m.r_ksath[s], inv_d);
  const double effk_avg = 0.5 * (effk_l + effk_r);
  F[(left ? LEFT_AQUIF2AQUIF : RIGHT_AQUIF2AQUIF) * nr + s] =
      sub_elem_to_river(gw_e, zmin_e, effk_e, r, effk_avg, inv_d);
}

// part-major, each part's segments padded to whole warps
__global__ void __launch_bounds__(128) k_river(DevMesh m, const double *RESTRICT y) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int pad = (m.nr_run + 31) & ~31;
  const int part = t / pad, s = t - part * pad;
  int sy;
  if (part >= kRivParts || s >= m.nr_run || skip_item(m, m.sys_riv, s, &sy)) return;
  river_part(m, y, s, part);
}

// ---------------------------------------------------------------------------
// k_river_rows: upstream sums and the river rows of ydot
// ---------------------------------------------------------------------------
// What a river row reads of the mesh: the first upstream segments' indices
// are a chain of loads in front of their fluxes.
struct RiverRowsIn {
  double area, porosity;
  int first, end, up[3];
};
__device__ __forceinline__ RiverRowsIn river_rows_load(const DevMesh &m, int s) {
  RiverRowsIn r;
  r.area = m.r_area[s];
  r.porosity = m.r_porosity[s];
  r.first = m.up_ptr[s];
  r.end = m.up_end[s];
#pragma unroll
  for (int k = 0; k < 3; k++) r.up[k] = r.first + k < r.end ? m.up_idx[r.first + k] : 0;
  return r;
}

// the quotients of a row, beside each other
__device__ __forceinline__ void river_rows_item(const DevMesh &m, double *ydot, int s, int sy, const RiverRowsIn &r) {
  const int nr = m.nr, ne = m.ne;
  const double *F = m.rivflow;
  double f[7];
  f[0] = F[UP_CHANL2CHANL * nr + s];
#pragma unroll
  for (int j = 1; j <= 6; j++) f[j] = F[j * nr + s];
  const double aq_l = F[LEFT_AQUIF2AQUIF * nr + s], aq_r = F[RIGHT_AQUIF2AQUIF * nr + s];
  const double aq_d = F[DOWN_AQUIF2AQUIF * nr + s];
  const double area = r.area, por_area = r.porosity * area;
  double up_c = f[0];
  double up_a = 0.0;
  double fc[3], fa[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    fc[k] = F[DOWN_CHANL2CHANL * nr + r.up[k]];
    fa[k] = F[DOWN_AQUIF2AQUIF * nr + r.up[k]];
  }
#pragma unroll
  for (int k = 0; k < 3; k++)
    if (r.first + k < r.end) {
      up_c -= fc[k];
      up_a -= fa[k];
    }
  for (int k = r.first + 3; k < r.end; k++) {
    const int u = m.up_idx[k];
    up_c -= F[DOWN_CHANL2CHANL * nr + u];
    up_a -= F[DOWN_AQUIF2AQUIF * nr + u];
  }
  f[0] = up_c;
  double dg = -aq_l - aq_r - aq_d - up_a + f[CHANL_LKG];
  double q[7], qg;
  bool ok = im::div_i(dg, por_area, qg);
#pragma unroll
  for (int j = 0; j <= 6; j++) ok &= im::div_i(f[j], area, q[j]);
  if (!ok) {
    qg = div_any(dg, por_area);
#pragma unroll
    for (int j = 0; j <= 6; j++) q[j] = div_any(f[j], area);
  }
  dg = qg;
  double ds = 0.0;
#pragma unroll
  for (int j = 0; j <= 6; j++) ds -= q[j];
  ydot[3 * ne + s] = ds;
  ydot[3 * ne + nr + s] = dg;
  if (m.diag) {
    m.rivflow[UP_CHANL2CHANL * nr + s] = up_c;
    m.rivflow[UP_AQUIF2AQUIF * nr + s] = up_a;
  }
  if (cmp::isnan_(ds) | cmp::isnan_(dg)) report_err(m, sy);
}

__global__ void __launch_bounds__(128) k_river_rows(DevMesh m, double *RESTRICT ydot) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  int sy;
  if (s >= m.nr_run || skip_item(m, m.sys_riv, s, &sy)) return;
  river_rows_item(m, ydot, s, sy, river_rows_load(m, s));
}

// kFromRef: the host-buffer evaluation, where the state arrives in reference
// order in memory the device reads over the host link.  Thread r then takes
// reference element r (the link read is contiguous), stores its three values
// at the element's internal position in y_int and prepares that element; the
// threads past the elements copy the river values.  This replaces a separate
// reordering pass, and the preparation runs under the transfer.
template <bool kFromRef>
__global__ void __launch_bounds__(kPrepBlock) k_elem_prep(DevMesh m, const double *y, const double *y_ref,
                                                          double *RESTRICT y_int, const int32_t *RESTRICT iperm,
                                                          int river_blocks) {
  __shared__ int qs_i[kPrepBlock], qd_i[kPrepBlock];
  __shared__ double qs_x[kPrepBlock], qd_num[kPrepBlock], qd_den[kPrepBlock];
  __shared__ int qs_n, qd_n;
  int sy = 0;
  // With more blocks than the SMs hold at once (8 each), k_elem_grad's would
  // stand waiting through the last of them: its blocks come when these end.
  // Eight evaluations of 400,000 elements: on four streams that fill the
  // device 1,035 us, 1,053 with the early start; on two 1,060 and 1,055, and
  // one evaluation with its reordering 154 and 153.  In one wave the early
  // start gives 4 us of 86.
  const bool early = gridDim.x <= kPrepWave;
  wait_for_previous();
  if (early || (int)blockIdx.x < river_blocks) next_may_start();
  if ((int)blockIdx.x < river_blocks) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < m.nr_run && !skip_item(m, m.sys_riv, s, &sy)) geom_item(m, kFromRef ? y_ref : y, s);
    return;
  }
  if (threadIdx.x == 0) {
    qs_n = 0;
    qd_n = 0;
  }
  __syncthreads();
  const int t0 = (blockIdx.x - river_blocks) * blockDim.x + threadIdx.x;
  int i = t0;
  double y_surf = 0.0, y_gw = 0.0;
  bool elem;
  if (kFromRef) {
    const int ne = m.ne;
    elem = t0 < ne;
    if (elem) {
      i = iperm[t0];
      y_surf = y_ref[t0];
      const double u = y_ref[ne + t0];
      y_gw = y_ref[2 * ne + t0];
      y_int[i] = y_surf;
      y_int[ne + i] = u;
      y_int[2 * ne + i] = y_gw;
    } else if (t0 < ne + 2 * m.nr) {
      y_int[2 * ne + t0] = y_ref[2 * ne + t0];  // stage and river gw, same order
    }
  } else {
    elem = i < m.ne_run && !skip_item(m, m.sys_elem, i, &sy);
    if (elem) {
      y_surf = y[i];
      y_gw = y[2 * m.ne + i];
    }
  }
  bool thin = false, mix = false;
  double sx = 0.0, num = 0.0, den = 0.0;
  if (elem) prep_item(m, i, y_surf, y_gw, thin, sx, mix, num, den);
  if (!early) next_may_start();
  const int ss = queue_slot(&qs_n, thin);
  if (thin) {
    qs_i[ss] = i;
    qs_x[ss] = sx;
  }
  const int sd = queue_slot(&qd_n, mix);
  if (mix) {
    qd_i[sd] = i;
    qd_num[sd] = num;
    qd_den[sd] = den;
  }
  __syncthreads();
  const int t = threadIdx.x;
  if (t < qs_n) prep_root(m, qs_i[t], qs_x[t]);
  if (t < qd_n) m.effk[qd_i[t]] = div_any(qd_num[t], qd_den[t]);
}

// ---------------------------------------------------------------------------
// k_elem_grad
// ---------------------------------------------------------------------------
// What the gradient reads besides the elements' heads: the element whose head
// each side takes (its own at a no-flow boundary), or -1 and the head itself
// (a river's water level, a boundary value); and the geometry.
struct GradIn {
  int32_t src[3];
  double h[3], x[3], y[3], inv_x, inv_y;
};
__device__ __forceinline__ GradIn grad_load(const DevMesh &m, const double *y, int i) {
  const int ne = m.ne;
  GradIn g;
#pragma unroll
  for (int j = 0; j < 3; j++) {
    g.src[j] = m.nb[j * ne + i];
    g.x[j] = m.nabr_x[j * ne + i];
    g.y[j] = m.nabr_y[j * ne + i];
    g.h[j] = 0.0;
  }
  g.inv_x = m.inv_den_x[i];
  g.inv_y = m.inv_den_y[i];
#pragma unroll
  for (int j = 0; j < 3; j++)
    if (g.src[j] < 0) {
      if (g.src[j] != kBoundary) {
        const int s = -1 - g.src[j];
        const double stage = clamp0(y[3 * ne + s]);
        g.h[j] = cmp::gt_v(stage, m.r_depth[s]) ? m.r_zbed[s] + stage : m.r_zmax[s];
        g.src[j] = -1;
      } else if (m.bctype[j * ne + i] == 0) {
        g.src[j] = i;
      } else {
        g.h[j] = m.elem_bc[j * ne + i];
        g.src[j] = -1;
      }
    }
  return g;
}
__device__ __forceinline__ double grad_value(const DevMesh &m, const GradIn &g) {
  double h[3];
#pragma unroll
  for (int j = 0; j < 3; j++) h[j] = g.src[j] >= 0 ? m.head[g.src[j]] : g.h[j];
  const double y0 = g.y[0], y1 = g.y[1], y2 = g.y[2];
  const double x0 = g.x[0], x1 = g.x[1], x2 = g.x[2];
  // DhByDl(nabr_y, nabr_x, h) and DhByDl(nabr_x, nabr_y, h)
  const double dhdx = -1.0 * (y2 * (h[1] - h[0]) + y1 * (h[0] - h[2]) + y0 * (h[2] - h[1])) * g.inv_x;
  const double dhdy = -1.0 * (x2 * (h[1] - h[0]) + x1 * (h[0] - h[2]) + x0 * (h[2] - h[1])) * g.inv_y;
  return sqrt_any(dhdx * dhdx + dhdy * dhdy);
}

// (40 registers, the gradient's own need: the river fluxes' 50 would keep a
// sixth of the SM's warps out)
__global__ void __launch_bounds__(256, 6) k_elem_grad(DevMesh m, const double *y, int river_blocks, bool from_ref) {
  int sy;
  if ((int)blockIdx.x < river_blocks) {
    wait_for_previous();
    next_may_start();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int pad = (m.nr_run + 31) & ~31;
    const int part = t / pad, s = t - part * pad;
    if (part < kRivParts && s < m.nr_run && !skip_item(m, m.sys_riv, s, &sy)) river_part(m, y, s, part);
    return;
  }
  const int i = (blockIdx.x - river_blocks) * blockDim.x + threadIdx.x;
  const bool on = i < m.ne_run && !skip_item(m, m.sys_elem, i, &sy);
  GradIn g;
  if (on && !from_ref) g = grad_load(m, y, i);
  wait_for_previous();
  next_may_start();
  if (on && from_ref) g = grad_load(m, y, i);
  if (on) m.gradmag[i] = grad_value(m, g);
}

// ---------------------------------------------------------------------------
// k_edge: one thread per interior edge.  SubFlowElemToElem and
// OvlFlowElemToElem (src/lat_flow.c:285-338) are antisymmetric in IEEE
// arithmetic under the diffusion wave (negated head difference, commutative
// averages, the same distance and edge length on both sides, which the host
// checks bit for bit), so the owner evaluates each edge once and the
// neighbour reads the negated value.  Kinematic overland flow is not
// antisymmetric (avg_sf depends on the sign of the gradient): there every
// element side is its own one-sided edge.
//
// The Manning flux costs about 35 FP64 operations and only edges whose
// upwind element holds water above the depression storage have one (about
// half of them, spread over nearly every warp).  So each thread computes its
// Darcy flux and the Manning flux's inputs, the edges with water are queued
// in shared memory (warp-aggregated slots), and after one barrier the block
// evaluates the queue densely: ceil(n/32) warps instead of all eight carry
// the powers.  Each flux depends on its edge alone, so which thread computes
// it changes no bit.
// ---------------------------------------------------------------------------
constexpr int kEdgeBlock = 256;

// The Darcy flux of edge e (owner i, neighbour k), stored, and the Manning
// flux's depth and head difference; false (and a zero flux stored) when the
// upwind element holds no water above the depression storage.
__device__ __forceinline__ bool edge_item(const DevMesh &m, const double *y, int e, int i, int k, double &avg_h,
                                          double &diff_h) {
  const int ne = m.ne;
  // Darcy flux between the two groundwater columns,
  // avg_ksat grad_h avg_h edge = (effk_i + effk_k) diff_h avg_h edge/(2 dist)
  const double gw_i = clamp0(y[2 * ne + i]), gw_k = clamp0(y[2 * ne + k]);
  diff_h = (gw_i + m.zmin[i]) - (gw_k + m.zmin[k]);
  avg_h = avg_h_sub(diff_h, gw_i, gw_k);
  m.eflux_sub[e] = (m.effk[i] + m.effk[k]) * diff_h * avg_h * m.e_subk[e];
  // Manning overland flux, crossa h^p grad_h / (sqrt(avg_sf) avg_rough) =
  // avg_h h^p diff_h / sqrt(avg_sf) edge/(dist avg_rough)
  const double s_i = m.surfh[i], s_k = m.surfh[k];
  diff_h = m.surf_mode == kKinematic ? m.zmax[i] - m.zmax[k] : m.head[i] - m.head[k];
  avg_h = avg_h_surf(diff_h, s_i, s_k);
  // avg_h == 0 gives crossa == 0: the flux is zero
  const bool wet = cmp::gt0(avg_h);
  if (!wet) m.eflux_ovl[e] = 0.0;
  return wet;
}
// the friction slope of edge e
__device__ __forceinline__ double edge_slope(const DevMesh &m, int e, int i, int k, double diff_h) {
  if (m.surf_mode == kKinematic) {
    const double grad_h = diff_h * m.e_invdist[e];
    return cmp::gt0(grad_h) ? grad_h : kGradMin;
  }
  const double avg_sf = 0.5 * (m.gradmag[i] + m.gradmag[k]);
  return cmp::gt_c(avg_sf, kGradMin) ? avg_sf : kGradMin;
}
__device__ __forceinline__ double edge_hp(double h) { return h * pow_manning(h, kManningSurf); }

__global__ void __launch_bounds__(kEdgeBlock) k_edge(DevMesh m, const double *y) {
  __shared__ int q_e[kEdgeBlock];
  __shared__ double q_h[kEdgeBlock], q_d[kEdgeBlock], q_sf[kEdgeBlock];
  __shared__ int q_n;
  if (threadIdx.x == 0) q_n = 0;
  __syncthreads();
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  int sy;
  bool wet = false;
  double avg_h = 0.0, diff_h = 0.0, avg_sf = 0.0;
  int i = 0, k = 0;
  const bool on = e < m.nedge_run && !skip_item(m, m.sys_edge, e, &sy);
  if (on) {
    i = m.e_i[e];
    k = m.e_k[e];
  }
  wait_for_previous();
  next_may_start();
  if (on) {
    wet = edge_item(m, y, e, i, k, avg_h, diff_h);
    avg_sf = edge_slope(m, e, i, k, diff_h);
  }
  const int slot = queue_slot(&q_n, wet);
  if (wet) {
    q_e[slot] = e;
    q_h[slot] = avg_h;
    q_d[slot] = diff_h;
    q_sf[slot] = avg_sf;
  }
  __syncthreads();
  const int t = threadIdx.x;
  if (t < q_n) {
    const int qe = q_e[t];
    m.eflux_ovl[qe] = edge_hp(q_h[t]) * q_d[t] * rsqrt(q_sf[t]) * m.e_ovlk[qe];
  }
}

// ---------------------------------------------------------------------------
// k_elem_main
// ---------------------------------------------------------------------------
// Block shapes: the same 64-register budget (1,024 resident threads per
// SM) cut into 512 x 2, 256 x 4 or 128 x 8 blocks.  With the elements
// ranked by branch class per block, 256 x 4 is fastest on large meshes (92
// against 102 and 97 us per 400k elements): larger blocks group more
// elements of a class but gather their loads from a wider window.  On a
// small mesh or a sparsely occupied batch arena the smaller blocks spread
// the work over more SMs.  The batch engine tunes the shape per arena.
//
// Branch classes: a block first sorts its elements by the branches the
// element rows take -- water table within the infiltration depth (no
// Psi/KrFunc, Recharge = Infil), ponded surface (EffKinf's second case),
// unsaturated zone deeper than the macropores (AvgKv's first case) -- so
// that a warp's lanes mostly take the same ones, and each thread then
// evaluates the element at its rank.  The classes only group; every element
// is evaluated by the same code whatever its class, so the results do not
// depend on the grouping.  Items that sit out (past the end, or a batch
// watershed without an evaluation) sort last and leave as whole warps.
constexpr int kElemClasses = 8;

__device__ __forceinline__ int elem_class(const DevMesh &m, const double *y, int i) {
  const int ne = m.ne;
  const double gw = clamp0(y[2 * ne + i]);
  const int ponded = cmp::gt_c(clamp0(y[i]), 0.5 * kDeprStg) ? 1 : 0;  // SurfH above the depression storage
  if (cmp::gt_v(gw, m.d_dinf[i])) return 4 + ponded;
  return 2 * ponded + (cmp::lt_v(gw, m.d_dmac[i]) ? 1 : 0);
}

// One element's rows, in three parts by what they wait for: the state alone
// (column_state), k_elem_prep's surface water (column_surface), the lateral
// fluxes (column_rows).  k_elem_main runs them in a row; k_rhs_fused runs the
// first two while other blocks work on the lateral fluxes.
struct Column {
  double gw, unsat, depth, rechg;                 // rechg: unless in_dinf, then infil's
  double satn_i, satk_i, psi_i, sq_i;             // Infil's saturation, KrFunc, Psi, its root
  double surfh, dh_by_dz;
  double kinf_crack;                              // EffKinf with the cracks partly filled (kCrack)
  double edir_surf, edir_unsat, edir_gw, ett_unsat, ett_gw;
  bool in_dinf, full, noah;                       // water table within dinf; no room left; Flux-PIHM
};

__device__ __forceinline__ void column_state(const DevMesh &m, const double *y, int i, int sy, Column &c) {
  const int ne = m.ne;
  const double gw = clamp0(y[2 * ne + i]);
  const double unsat = clamp0(y[ne + i]);
  // The saturation's powers first: they are the register-hungry part, and
  // nothing else of the element is live while they run (with the edge fluxes
  // and the column's parameters loaded before them, 64 registers spilled
  // 330 bytes a thread).
  const double depth = m.depth[i];
  const bool gw_in_dinf = cmp::gt_v(gw, m.d_dinf[i]);
  c.noah = m.noah && (!m.sys_noah || m.sys_noah[sy]);
  c.gw = gw;
  c.unsat = unsat;
  c.depth = depth;
  c.in_dinf = gw_in_dinf;
  c.full = cmp::gt_v(unsat + gw, depth);
  // KrFunc(beta, 1) == 1 exactly: pow(1 - pow(1, m), e) == pow(0, e) == 0
  double satn = 1.0, satkfunc = 1.0, psi_u = 0.0, sq = 1.0;
  c.rechg = 0.0;
  if (!gw_in_dinf) {
    const double deficit = depth - gw;
    satn = div_any(unsat, deficit);
    satn = cmp::gt_c(satn, 1.0) ? 1.0 : satn;
    satn = cmp::lt_c(satn, kSatMin) ? kSatMin : satn;
    kr_psi(satn, m.vg_m[i], m.vg_e[i], m.vg_ib[i], m.alpha[i], satkfunc, psi_u, sq);
    // Recharge, src/vert_flow.c:132-170: the denominators add up to depth
    // ((deficit + gw) and the AvgKv weights d1 + d2 + d3, to an ulp);
    // multiply by 1/depth instead
    const double inv_depth = m.inv_depth[i], ksatv = m.ksatv[i], dmac = m.dmac[i];
    const double dh_by_dz = (0.5 * deficit + psi_u) * (2.0 * inv_depth);
    // AvgKv, src/vert_flow.c:172-209, arithmetic mean (_ARITH_ is defined at
    // src/include/pihm_func.h:4)
    double k1, k2, k3, d1, d2, d3;
    if (cmp::gt_v(deficit, dmac)) {
      k1 = satkfunc * ksatv;
      d1 = dmac;
      k2 = satkfunc * ksatv;
      d2 = deficit - dmac;
      k3 = ksatv;
      d3 = gw;
    } else {
      k1 = satkfunc * ksatv;
      d1 = deficit;
      k2 = m.kv2_mac[i];
      d2 = dmac - deficit;
      k3 = ksatv;
      d3 = gw - (dmac - deficit);
    }
    const double kavg = (k1 * d1 + k2 * d2 + k3 * d3) * inv_depth;
    double rechg = kavg * dh_by_dz;
    rechg = (cmp::gt0(rechg) && cmp::le0(unsat)) ? 0.0 : rechg;
    rechg = (cmp::lt0(rechg) && cmp::le0(gw)) ? 0.0 : rechg;
    c.rechg = rechg;
  }
  // Infil's saturation: the same one, except in Flux-PIHM, where it is
  // Noah's top-layer moisture (src/vert_flow.c:94-98) and Recharge keeps
  // the column's
  c.satn_i = satn;
  c.satk_i = satkfunc;
  c.psi_i = psi_u;
  c.sq_i = sq;
  if (c.noah && !gw_in_dinf) {
    double s = m.noah_satn[i];
    s = cmp::gt_c(s, 1.0) ? 1.0 : s;
    s = cmp::lt_c(s, kSatMin) ? kSatMin : s;
    c.satn_i = s;
    kr_psi(s, m.vg_m[i], m.vg_e[i], m.vg_ib[i], m.alpha[i], c.satk_i, c.psi_i, c.sq_i);
  }
}

// EffKinf's conductivity where the cracks carry part of their flow
// (src/vert_flow.c:211-270).  KrFunc(2, satn): pow(satn, 2) and pow(., 0.5)
// are a product and sqrt; the root of the saturation is kr_psi's (1 where it
// is 1).  The roundings are spelt out: every kernel that inlines this
// rounds alike.
__device__ __forceinline__ double crack_kinf(const Column &c, double kinf_mat, double kmac_a) {
  const double t2 = 1.0 - sqrt_any(fma(-c.satn_i, c.satn_i, 1.0));
  return fma(kmac_a, __dmul_rn(__dmul_rn(c.sq_i, t2), t2), __dmul_rn(kinf_mat, c.satk_i));
}

__device__ __forceinline__ void column_surface(const DevMesh &m, int i, Column &c) {
  const double surfh = m.surfh[i];
  c.surfh = surfh;
  // Infil's head gradient, src/vert_flow.c:33-130
  c.dh_by_dz = 0.0;
  if (!c.full) {
    const double zmax = m.zmax[i];
    const double dinf = m.dinf[i];
    // the head below the infiltration front: the water table when it lies
    // within dinf of the surface, else the unsaturated zone's; both
    // reference branches divide (surfh + zmax - head) by the same
    // denominator, so one division serves a warp whose lanes take both
    double h_u = c.gw + m.zmin[i];
    if (!c.in_dinf) {
      const double psi_c = cmp::gt_nc(c.psi_i, kPsiMin) ? c.psi_i : kPsiMin;
      h_u = psi_c + zmax - 0.5 * dinf;
    }
    const double dh_by_dz = div_any(surfh + zmax - h_u, 0.5 * (surfh + dinf));
    c.dh_by_dz = (cmp::le0(surfh) && cmp::gt0(dh_by_dz)) ? 0.0 : dh_by_dz;
  }
  // EtExtract, src/hydrol.c:33-97
  const double edir = m.edir[i], ett = m.ett[i];
  c.edir_surf = c.edir_unsat = c.edir_gw = c.ett_unsat = c.ett_gw = 0.0;
  if (c.noah) {
    // Flux-PIHM (src/hydrol.c:43-55,79-83): no ponded-water source, and the
    // transpiration split by GwTransp (noah/lsm_func.c:163-185) over the
    // Noah layers from the water table down to the root depth
    if (c.in_dinf) c.edir_gw = edir;
    else c.edir_unsat = edir;
    double gwet = 0.0;
    if (cmp::gt0(ett) && m.noah_wtin[i]) {
      gwet = div_any(m.noah_etgw[i], ett);
      gwet = cmp::gt_c(gwet, 1.0) ? 1.0 : gwet;
      gwet = cmp::lt0(gwet) ? 0.0 : gwet;
    }
    c.ett_unsat = (1.0 - gwet) * ett;
    c.ett_gw = gwet * ett;
  } else {
    if (cmp::ge_c(surfh, kDeprStg)) c.edir_surf = edir;
    else if (c.in_dinf) c.edir_gw = edir;
    else c.edir_unsat = edir;
    if (cmp::gt_v(c.gw, m.d_rzd[i])) c.ett_gw = ett;
    else c.ett_unsat = ett;
  }
}

// The element's parameters that the rows read, and where its lateral fluxes
// are.  riv[j]: the river segment of side j, or -1; right[j]: its right bank.
// ovl[j]: on river edges the previous evaluation's flux, which Infil sees.
struct RowsIn {
  int32_t code[3], riv[3];
  bool right[3];
  double ovl[3];
  double inv_area, inv_por, pcpdrp, ws0, kinf_mat, kmac_a, areafh, kinfv;
};
__device__ __forceinline__ void rows_load(const DevMesh &m, int i, RowsIn &r) {
  const int ne = m.ne;
#pragma unroll
  for (int j = 0; j < 3; j++) {
    r.code[j] = m.emap[j * ne + i];
    r.riv[j] = -1;
    r.right[j] = false;
    r.ovl[j] = 0.0;
  }
  r.inv_area = m.inv_area[i];
  r.inv_por = m.inv_por[i];
  r.pcpdrp = m.pcpdrp[i];
  r.ws0 = m.ws0_surf[i];
  r.kinf_mat = m.kinf_mat[i];
  r.kmac_a = m.kmac_a[i];
  r.areafh = m.areafh[i];
  r.kinfv = m.kinfv[i];
  if (r.code[0] == 0 || r.code[1] == 0 || r.code[2] == 0) {
    int32_t nb[3];
#pragma unroll
    for (int j = 0; j < 3; j++) nb[j] = m.nb[j * ne + i];
#pragma unroll
    for (int j = 0; j < 3; j++) r.riv[j] = (r.code[j] == 0 && nb[j] < 0 && nb[j] != kBoundary) ? -1 - nb[j] : -1;
#pragma unroll
    for (int j = 0; j < 3; j++)
      if (r.riv[j] >= 0) r.right[j] = m.left[r.riv[j]] != i;
#pragma unroll
    for (int j = 0; j < 3; j++)
      if (r.riv[j] >= 0) r.ovl[j] = -m.carry_ovl[(r.right[j] ? m.nr : 0) + r.riv[j]];
  }
}

// kBanks: this evaluation's river fluxes are done, so an element with river
// edges finishes its rows here; otherwise it hands its partial sums to
// k_bank_rows.
template <bool kBanks>
__device__ __forceinline__ void column_rows(const DevMesh &m, double *ydot, int i, int sy, const Column &c,
                                            const RowsIn &r) {
  const int ne = m.ne;
  const double surfh = c.surfh, inv_area = r.inv_area, pcpdrp = r.pcpdrp;
  // edge fluxes, with the sign seen from this element (a negative code: the
  // flux was computed from the neighbour's side); 0 on domain boundaries
  // (BoundFluxElem)
  double ovl[3], sub[3], f[3][3];
  bool riv[3];
#pragma unroll
  for (int j = 0; j < 3; j++) {
    const int32_t code = r.code[j];
    riv[j] = r.riv[j] >= 0;
    ovl[j] = r.ovl[j];
    sub[j] = 0.0;
    if (code != 0) ovl[j] = cmp::neg_if(m.eflux_ovl[(code > 0 ? code : -code) - 1], code < 0);
    // (kBanks: every load of this side now, so that they are in flight together)
    if (kBanks && code != 0) sub[j] = m.eflux_sub[(code > 0 ? code : -code) - 1];
  }
  if (kBanks && (riv[0] || riv[1] || riv[2])) {
    const double *F = m.rivflow;
    const int nr = m.nr;
#pragma unroll
    for (int j = 0; j < 3; j++)
      if (riv[j]) {
        f[j][0] = F[(r.right[j] ? RIGHT_SURF2CHANL : LEFT_SURF2CHANL) * nr + r.riv[j]];
        f[j][1] = F[(r.right[j] ? RIGHT_AQUIF2CHANL : LEFT_AQUIF2CHANL) * nr + r.riv[j]];
        f[j][2] = F[(r.right[j] ? RIGHT_AQUIF2AQUIF : LEFT_AQUIF2AQUIF) * nr + r.riv[j]];
      }
  }
  const double edir_surf = c.edir_surf, edir_unsat = c.edir_unsat, edir_gw = c.edir_gw;
  const double ett_unsat = c.ett_unsat, ett_gw = c.ett_gw;

  // Infil, src/vert_flow.c:33-130
  double infil;
  if (c.full) {
    infil = 0.0;
  } else {
    const double dh_by_dz = c.dh_by_dz;
    double applrate = 0.0;
#pragma unroll
    for (int j = 0; j < 3; j++) applrate += -ovl[j] * inv_area;
    applrate = cmp::gt0(applrate) ? applrate : 0.0;
    applrate += pcpdrp;
    double wetfrac = surfh * (1.0 / kDeprStg);
    wetfrac = cmp::gt0(wetfrac) ? wetfrac : 0.0;
    wetfrac = cmp::lt_c(wetfrac, 1.0) ? wetfrac : 1.0;
    // EffKinf, src/vert_flow.c:211-270 (its roundings spelt out, as in
    // crack_kinf)
    const double mat = __dmul_rn(r.kinf_mat, c.satk_i);
    const double both = __dadd_rn(mat, r.kmac_a);
    double kinf;
    if (cmp::eq0(r.areafh)) {
      kinf = r.kinfv * c.satk_i;
    } else if (cmp::gt_c(surfh, kDeprStg)) {
      kinf = fma(r.kinf_mat, c.satk_i, r.kmac_a);
    } else if (cmp::le_v(applrate, dh_by_dz * r.kinfv * c.satk_i)) {
      kinf = r.kinfv * c.satk_i;
    } else if (cmp::lt_v(applrate, dh_by_dz * both)) {
      kinf = kBanks ? c.kinf_crack : crack_kinf(c, r.kinf_mat, r.kmac_a);
    } else {
      kinf = both;
    }
    infil = kinf * dh_by_dz;
    if (!c.in_dinf) infil = cmp::gt0(infil) ? infil : 0.0;
    const double ws0 = r.ws0;
    const double inv_dt = m.sys_inv_dt ? m.sys_inv_dt[sy] : m.inv_dt;
    const double infil_max = applrate + (cmp::gt0(ws0) ? ws0 * inv_dt : 0.0);
    infil = cmp::gt_v(infil, infil_max) ? infil_max : infil;
    infil *= wetfrac;
  }
  if (c.noah) infil *= m.noah_fcr[i];  // frozen top soil, src/vert_flow.c:16-19
  const double rechg = c.in_dinf ? infil : c.rechg;

  // groundwater fluxes
#pragma unroll
  for (int j = 0; j < 3; j++) {
    const int32_t code = r.code[j];
    if (code != 0) {
      sub[j] = cmp::neg_if(kBanks ? sub[j] : m.eflux_sub[(code > 0 ? code : -code) - 1], code < 0);
    } else if (!riv[j]) {
      // BoundFluxElem, src/lat_flow.c:340-382
      const int bct = m.bctype[j * ne + i];
      if (bct > 0) {
        const double bc = m.elem_bc[j * ne + i], zmin = m.zmin[i];
        const double diff_h = c.gw + zmin - bc;
        const double avg_h = avg_h_sub(diff_h, c.gw, bc - zmin);
        const double grad_h = div_any(diff_h, m.nabrdist[j * ne + i]);
        sub[j] = m.effk[i] * grad_h * avg_h * m.edge[j * ne + i];
      } else if (bct < 0) {
        sub[j] = -m.elem_bc[j * ne + i];
      }
    }
  }

  if (m.diag) {
#pragma unroll
    for (int j = 0; j < 3; j++) {
      if (!riv[j]) {
        m.d_ovl[j * ne + i] = ovl[j];
        m.d_sub[j * ne + i] = sub[j];
      }
    }
    m.d_infil[i] = infil;
    m.d_rechg[i] = rechg;
    m.d_et[i] = edir_surf;
    m.d_et[ne + i] = edir_unsat;
    m.d_et[2 * ne + i] = edir_gw;
    m.d_et[3 * ne + i] = ett_unsat;
    m.d_et[4 * ne + i] = ett_gw;
  }

  // river edges: this evaluation's fluxes, and the overland one kept for the
  // next evaluation's Infil.  A bank's slot of carry_ovl is read in rows_load
  // and written here by its own element's thread alone.
  if (kBanks && (riv[0] || riv[1] || riv[2])) {
    const int nr = m.nr;
#pragma unroll
    for (int j = 0; j < 3; j++)
      if (riv[j]) {
        ovl[j] = -f[j][0];
        sub[j] = -(f[j][1] + f[j][2]);
        m.carry_ovl[(r.right[j] ? nr : 0) + r.riv[j]] = f[j][0];
        if (m.diag) {
          m.d_ovl[j * ne + i] = ovl[j];
          m.d_sub[j * ne + i] = sub[j];
        }
      }
  }

  // element rows of ydot, src/ode.c:111-209
  const double inv_por = r.inv_por;
  const double base_surf = pcpdrp - infil - edir_surf;
  const double base_gw = rechg - edir_gw - ett_gw;
  const double du = (infil - rechg - edir_unsat - ett_unsat) * inv_por;
  ydot[ne + i] = du;
  unsigned int bad = cmp::isnan_(du);
  if (!kBanks && (riv[0] || riv[1] || riv[2])) {
    const int b = m.bank_slot[i];
    const int nbk = m.nbank;
    double *bp = m.bank_part;
    bp[b] = base_surf;
    bp[nbk + b] = base_gw;
#pragma unroll
    for (int j = 0; j < 3; j++) {
      bp[(2 + j) * nbk + b] = ovl[j];
      bp[(5 + j) * nbk + b] = sub[j];
    }
    if (bad) report_err(m, sy);
    return;
  }
  double ds = base_surf, dg = base_gw;
#pragma unroll
  for (int j = 0; j < 3; j++) {
    ds -= ovl[j] * inv_area;
    dg -= sub[j] * inv_area;
  }
  dg *= inv_por;
  ydot[i] = ds;
  ydot[2 * ne + i] = dg;
  bad |= cmp::isnan_(ds) | cmp::isnan_(dg);
  if (bad) report_err(m, sy);
}

template <int BLOCK, int MINB>
__global__ void __launch_bounds__(BLOCK, MINB) k_elem_main(DevMesh m, const double *y, double *RESTRICT ydot,
                                                           bool from_ref) {
  // the state itself may be read before the kernels ahead have finished,
  // unless they wrote it
  if (from_ref) wait_for_previous();
  // a stable ranking: class-major, then warp, then lane, so each class keeps
  // the block's element order and a warp's elements lie close together
  constexpr int kWarps = BLOCK / 32, kSlots = kElemClasses * kWarps;
  __shared__ int s_off[kSlots];  // [class][warp]: count, then exclusive offset
  __shared__ unsigned short s_order[BLOCK];
  {
    const int i0 = blockIdx.x * BLOCK + threadIdx.x;
    int sy0;
    const int cls = (i0 >= m.ne_run || skip_item(m, m.sys_elem, i0, &sy0)) ? kElemClasses - 1
                                                                          : elem_class(m, y, i0);
    for (int k = threadIdx.x; k < kSlots; k += BLOCK) s_off[k] = 0;
    __syncthreads();
    const unsigned lane = threadIdx.x & 31u;
    const int warp = threadIdx.x >> 5;
    const unsigned peers = __match_any_sync(0xffffffffu, cls);
    if ((int)lane == __ffs(peers) - 1) s_off[cls * kWarps + warp] = __popc(peers);
    __syncthreads();
    if (warp == 0) {
      // exclusive scan of the kSlots counts: each lane sums its run of
      // consecutive slots, the lanes scan their sums, then write back
      constexpr int kRun = (kSlots + 31) / 32;
      int run[kRun], sum = 0;
#pragma unroll
      for (int r = 0; r < kRun; r++) {
        const int k = (int)lane * kRun + r;
        run[r] = k < kSlots ? s_off[k] : 0;
        sum += run[r];
      }
      int incl = sum;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, d);
        if ((int)lane >= d) incl += v;
      }
      int off = incl - sum;
#pragma unroll
      for (int r = 0; r < kRun; r++) {
        const int k = (int)lane * kRun + r;
        if (k < kSlots) s_off[k] = off;
        off += run[r];
      }
    }
    __syncthreads();
    s_order[s_off[cls * kWarps + warp] + __popc(peers & ((1u << lane) - 1u))] = (unsigned short)threadIdx.x;
    __syncthreads();
  }
  const int i = blockIdx.x * BLOCK + s_order[threadIdx.x];
  int sy;
  const bool on = i < m.ne_run && !skip_item(m, m.sys_elem, i, &sy);
  Column c;
  if (on) column_state(m, y, i, sy, c);
  wait_for_previous();
  next_may_start();
  if (!on) return;
  column_surface(m, i, c);
  RowsIn r;
  rows_load(m, i, r);
  column_rows<false>(m, ydot, i, sy, c, r);
}

// ---------------------------------------------------------------------------
// k_bank_rows: the rows of elements with river edges, from k_elem_main's
// partial sums and the river fluxes, and the overland flux kept for the next
// evaluation's Infil; and the river rows.  A chain of four dependent loads
// for a few thousand items: the three that lead to the fluxes (the element,
// its neighbours, the bank's side) are done while k_elem_main ends.
// ---------------------------------------------------------------------------
// (80 registers: its blocks stand in the SMs while k_elem_main ends; at 128 an
// ensemble of four contexts' 400,000 elements took 1,072 us instead of 1,058)
__global__ void __launch_bounds__(128, 6) k_bank_rows(DevMesh m, double *RESTRICT ydot, int river_blocks) {
  int sy;
  if ((int)blockIdx.x < river_blocks) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    const bool on = s < m.nr_run && !skip_item(m, m.sys_riv, s, &sy);
    RiverRowsIn in;
    if (on) in = river_rows_load(m, s);
    wait_for_previous();
    if (on) river_rows_item(m, ydot, s, sy, in);
    return;
  }
  const int b = (blockIdx.x - river_blocks) * blockDim.x + threadIdx.x;
  const bool on = b < m.nbank_run && !skip_item(m, m.sys_bank, b, &sy);
  const int nr = m.nr, ne = m.ne, nbk = m.nbank;
  int i = 0, seg[3] = {-1, -1, -1};
  bool left[3] = {false, false, false};
  double inv_area = 0.0, inv_por = 0.0;
  if (on) {
    i = m.bank_elem[b];
    inv_area = m.inv_area[i];
    inv_por = m.inv_por[i];
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const int32_t nb = m.nb[j * ne + i];
      if (nb < 0 && nb != kBoundary) {
        seg[j] = -1 - nb;
        left[j] = m.left[seg[j]] == i;
      }
    }
  }
  wait_for_previous();
  if (!on) return;
  const double *F = m.rivflow;
  const double *bp = m.bank_part;
  double ds = bp[b], dg = bp[nbk + b], f[3][3], o[3], u[3];
#pragma unroll
  for (int j = 0; j < 3; j++) {
    if (seg[j] >= 0) {
      f[j][0] = F[(left[j] ? LEFT_SURF2CHANL : RIGHT_SURF2CHANL) * nr + seg[j]];
      f[j][1] = F[(left[j] ? LEFT_AQUIF2CHANL : RIGHT_AQUIF2CHANL) * nr + seg[j]];
      f[j][2] = F[(left[j] ? LEFT_AQUIF2AQUIF : RIGHT_AQUIF2AQUIF) * nr + seg[j]];
    } else {
      o[j] = bp[(2 + j) * nbk + b];
      u[j] = bp[(5 + j) * nbk + b];
    }
  }
#pragma unroll
  for (int j = 0; j < 3; j++) {
    if (seg[j] >= 0) {
      o[j] = -f[j][0];
      u[j] = -(f[j][1] + f[j][2]);
      m.carry_ovl[(left[j] ? 0 : nr) + seg[j]] = f[j][0];
      if (m.diag) {
        m.d_ovl[j * ne + i] = o[j];
        m.d_sub[j * ne + i] = u[j];
      }
    }
    ds -= o[j] * inv_area;
    dg -= u[j] * inv_area;
  }
  dg *= inv_por;
  ydot[i] = ds;
  ydot[2 * ne + i] = dg;
  if (cmp::isnan_(ds) | cmp::isnan_(dg)) report_err(m, sy);
}

// ---------------------------------------------------------------------------
// k_rhs_fused: the whole evaluation in one cooperative launch, for meshes
// whose evaluation is the latency of dependent kernels.  The arithmetic of
// the kernels above, cut by what it depends on and given to four kinds of
// blocks that run beside each other:
//
//   elements  prep -> | A, heads -> gradient -> | B
//   edges             | A, Darcy flux, h^p ---- | B, slope -> flux | C
//   rivers    area, perimeter | R, channel flux ------------------- | C, rows
//   banks     area, perimeter | A, fluxes with the elements -------- (to C)
//   beds      area, perimeter | A, R, bed fluxes, outlets ---------- (to C)
//   columns   saturation, powers, recharge | A, infiltration's head | C, rows
//
// Everything a block can do without the others' results stands before its
// wait: an evaluation then takes the chain prep, gradient, slope, rows and
// three barriers, instead of seven kernels each with its own launch, loads
// and powers.  Each item's arithmetic is that of the separate kernels, so the
// results are the same bits.
//
// A, B, C, R are counters in device memory that the blocks before them raise
// once (R: every river block; C: edges, rivers, banks and beds).  The last
// block through C zeroes them -- every other block has raised C, or what C
// waits for, behind its own last wait -- so a captured launch can be replayed.
// For the elements' wait on A that holds because the edges wait for B: without
// an interior edge nothing would, so then (edges alone read the gradients) the
// elements are done when they have raised A.
// Cooperative launch makes the blocks resident together; a wait gives up after
// m.bar_polls polls, and the blocks then report kErrWait instead of results.
// ---------------------------------------------------------------------------
constexpr int kBarStride = 32;      // counters on cache lines of their own

__device__ __forceinline__ void bar_arrive(unsigned *cnt) {
  __syncthreads();
  if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(cnt) : "memory");
}
// false when the wait ran out; the same answer in every thread of the block
__device__ __forceinline__ bool bar_wait(const DevMesh &m, unsigned *cnt, unsigned blocks, int *s_ok) {
  if (threadIdx.x == 0) {
    unsigned v = 0;
    for (int k = 0; k < m.bar_polls; k++) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(cnt) : "memory");
      if (v >= blocks) break;
    }
    *s_ok = v >= blocks;
  }
  __syncthreads();
  const bool ok = *s_ok != 0;
  __syncthreads();
  return ok;
}

// a block is past its last wait: the last of `blocks` zeroes the counters
__device__ __forceinline__ void bar_leave(unsigned *bar, unsigned blocks) {
  if (threadIdx.x == 0 && atomicAdd(bar + 4 * kBarStride, 1u) == blocks - 1)
    for (int k = 0; k < 5; k++) bar[k * kBarStride] = 0u;
}

// what a block whose wait ran out leaves: the error word of its items
__device__ __noinline__ void report_wait(const DevMesh &m, const int32_t *sys_of, int first, int n, int step) {
  int sy;
  for (int k = first; k < n; k += step)
    if (!skip_item(m, sys_of, k, &sy)) report_err(m, sy, kErrWait);
}

constexpr int kFusedThreads = 256;  // most threads per block

// blocks of each kind, in this order of block index
struct FusedGrid {
  int elem, edge, river, col;
};

template <bool kFromRef, int kMinBlocks>
__global__ void __launch_bounds__(kFusedThreads, kMinBlocks)
    k_rhs_fused(const __grid_constant__ DevMesh m, const double *y, double *ydot, const double *y_ref, double *y_int,
                const int32_t *iperm, const FusedGrid g) {
  __shared__ int s_ok;
  unsigned *const A = m.bar, *const B = m.bar + kBarStride, *const C = m.bar + 2 * kBarStride,
                  *const R = m.bar + 3 * kBarStride;
  const bool grad = m.surf_mode == kDiffWave && g.edge > 0;
  const int ne = m.ne;
  int blk = blockIdx.x;
  int sy;
  wait_for_previous();
  if (blk < g.elem) {
    // ---- elements ----
    const int first = blk * blockDim.x + threadIdx.x, step = g.elem * blockDim.x;
    const int n = kFromRef ? ne + 2 * m.nr : m.ne_run;
    for (int t = first; t < n; t += step) {
      int i = t;
      double y_surf, y_gw;
      if (kFromRef) {
        if (t >= ne) {  // stage and river gw, same order
          y_int[2 * ne + t] = y_ref[2 * ne + t];
          continue;
        }
        i = iperm[t];
        y_surf = y_ref[t];
        const double u = y_ref[ne + t];
        y_gw = y_ref[2 * ne + t];
        y_int[i] = y_surf;
        y_int[ne + i] = u;
        y_int[2 * ne + i] = y_gw;
      } else {
        if (skip_item(m, m.sys_elem, i, &sy)) continue;
        y_surf = y[i];
        y_gw = y[2 * ne + i];
      }
      bool thin = false, mix = false;
      double sx, num, den;
      prep_item(m, i, y_surf, y_gw, thin, sx, mix, num, den);
      if (thin) prep_root(m, i, sx);
      if (mix) m.effk[i] = div_any(num, den);
    }
    bar_arrive(A);
    if (!grad) return;
    // kFromRef: the river stages grad_load reads are other blocks' copies
    const bool one = !kFromRef && step >= m.ne_run;  // one element a thread: its geometry before the wait
    const bool on = one && first < m.ne_run && !skip_item(m, m.sys_elem, first, &sy);
    GradIn in;
    if (on) in = grad_load(m, y, first);
    if (!bar_wait(m, A, g.elem, &s_ok)) return report_wait(m, m.sys_elem, first, m.ne_run, step);
    if (on) m.gradmag[first] = grad_value(m, in);
    for (int i = first; !one && i < m.ne_run; i += step)
      if (!skip_item(m, m.sys_elem, i, &sy)) m.gradmag[i] = grad_value(m, grad_load(m, y, i));
    bar_arrive(B);
    return;
  }
  blk -= g.elem;
  if (blk < g.edge) {
    // ---- edges ----
    const int first = blk * blockDim.x + threadIdx.x, step = g.edge * blockDim.x;
    if (!bar_wait(m, A, g.elem, &s_ok)) return report_wait(m, m.sys_edge, first, m.nedge_run, step);
    bool waited = !grad;
    // whole blocks go round together: the wait is the block's
    for (int e = first; e - (int)threadIdx.x < m.nedge_run; e += step) {
      int i = 0, k = 0;
      double avg_h = 0.0, diff_h = 0.0, hp = 0.0;
      bool wet = false;
      if (e < m.nedge_run && !skip_item(m, m.sys_edge, e, &sy)) {
        i = m.e_i[e];
        k = m.e_k[e];
        wet = edge_item(m, y, e, i, k, avg_h, diff_h);
        if (wet) hp = edge_hp(avg_h);
      }
      if (!waited) {
        waited = true;
        if (!bar_wait(m, B, g.elem, &s_ok)) return report_wait(m, m.sys_edge, first, m.nedge_run, step);
      }
      if (wet) m.eflux_ovl[e] = hp * diff_h * rsqrt(edge_slope(m, e, i, k, diff_h)) * m.e_ovlk[e];
    }
    bar_arrive(C);
    return;
  }
  blk -= g.edge;
  const unsigned lateral = g.edge + g.river;
  if (blk < g.river) {
    // ---- rivers: the same number of blocks for each part ----
    const int per = g.river / kRivParts, part = blk / per;
    const int first = (blk - part * per) * blockDim.x + threadIdx.x, step = per * blockDim.x;
    // areas and perimeters need the state alone; kFromRef: river values stand
    // in the same order.  Every part's blocks take a quarter of their
    // segments, so that no SM has a block full of them beside its elements
    // (21,000 elements: 9.5 us until the last with the channel blocks alone)
    const double *yr = kFromRef ? y_ref : y;
    const int quarter = blockDim.x / kRivParts;
    for (int s = first + part * quarter; s < m.nr_run; s += step)
      if ((int)threadIdx.x < quarter && !skip_item(m, m.sys_riv, s, &sy)) geom_item(m, yr, s);
    bar_arrive(R);
    bool ok;
    if (part == PART_CHAN) {
      ok = bar_wait(m, R, g.river, &s_ok);
      for (int s = first; ok && s < m.nr_run; s += step)
        if (!skip_item(m, m.sys_riv, s, &sy)) river_part(m, yr, s, PART_CHAN);
    } else {
      ok = bar_wait(m, A, g.elem, &s_ok);
      if (ok && part == PART_BED) ok = bar_wait(m, R, g.river, &s_ok);
      for (int s = first; ok && s < m.nr_run; s += step)
        if (!skip_item(m, m.sys_riv, s, &sy)) river_part(m, y, s, part);
    }
    if (ok) {
      bar_arrive(C);
      if (part != PART_CHAN) return;
    }
    const bool on = first < m.nr_run && !skip_item(m, m.sys_riv, first, &sy);
    RiverRowsIn in;
    if (on) in = river_rows_load(m, first);
    if (ok) ok = bar_wait(m, C, lateral, &s_ok);
    if (!ok) return report_wait(m, m.sys_riv, first, m.nr_run, step);
    bar_leave(m.bar, per + g.col);
    if (on) river_rows_item(m, ydot, first, sy, in);
    for (int s = first + step; s < m.nr_run; s += step)
      if (!skip_item(m, m.sys_riv, s, &sy)) river_rows_item(m, ydot, s, sy, river_rows_load(m, s));
    return;
  }
  blk -= g.river;
  // ---- columns ----
  const int first = blk * blockDim.x + threadIdx.x, step = g.col * blockDim.x;
  bool met = false;  // the block has been through A and C
  for (int i = first; i - (int)threadIdx.x < m.ne_run || !met; i += step) {
    const bool on = i < m.ne_run && !skip_item(m, m.sys_elem, i, &sy);
    Column c;
    RowsIn r;
    // kFromRef: the state in internal order is the element blocks' to write
    if (kFromRef && !met && !bar_wait(m, A, g.elem, &s_ok)) return report_wait(m, m.sys_elem, first, m.ne_run, step);
    if (on) {
      column_state(m, y, i, sy, c);
      rows_load(m, i, r);
    }
    if (!kFromRef && !met && !bar_wait(m, A, g.elem, &s_ok)) return report_wait(m, m.sys_elem, first, m.ne_run, step);
    if (on) {
      column_surface(m, i, c);
      c.kinf_crack = crack_kinf(c, r.kinf_mat, r.kmac_a);
    }
    if (!met) {
      met = true;
      if (!bar_wait(m, C, lateral, &s_ok)) return report_wait(m, m.sys_elem, first, m.ne_run, step);
      bar_leave(m.bar, g.river / kRivParts + g.col);
      }
    if (on) column_rows<true>(m, ydot, i, sy, c, r);
  }
}

// ---------------------------------------------------------------------------
// state reordering between reference and internal order
// ---------------------------------------------------------------------------
// blockIdx.y is the plane (surface, unsaturated, groundwater), and the blocks
// past its elements copy the river values; the index is read before the wait
// for the evaluation's last kernel (these are dependent launches too).
__global__ void __launch_bounds__(256) k_permute(const double *src, double *dst, const int32_t *RESTRICT perm, int ne,
                                                 int nr, int to_internal) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool elem = i < ne;
  const int r = elem ? perm[i] : 0;
  wait_for_previous();
  const long long plane = (long long)blockIdx.y * ne;
  if (elem) dst[plane + (to_internal ? i : r)] = src[plane + (to_internal ? r : i)];
  else if (blockIdx.y == 2 && i - ne < 2 * nr) dst[plane + i] = src[plane + i];
}

// The same reordering walked in reference order (iperm: reference ->
// internal element index): the reference-order side is read or written
// contiguously, which is the side in host memory when the host-buffer
// evaluation accesses it directly.
//
// With a status to hand over (done.host): the last block writes the error word
// and the sequence number behind every block's values, which saves the host
// call a kernel of its own for it.
__global__ void __launch_bounds__(256) k_permute_ref(const double *src, double *dst, const int32_t *RESTRICT iperm,
                                                     int ne, int nr, int to_internal, StatusOut done) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  const bool elem = r < ne;
  const int i = elem ? iperm[r] : 0;
  wait_for_previous();
  const long long plane = (long long)blockIdx.y * ne;
  if (elem) dst[plane + (to_internal ? i : r)] = src[plane + (to_internal ? r : i)];
  else if (blockIdx.y == 2 && r - ne < 2 * nr) dst[plane + r] = src[plane + r];
  if (!done.host) return;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence_system();
    if (atomicAdd(done.ticket, 1u) == gridDim.x * gridDim.y - 1) {
      *done.ticket = 0u;
      __threadfence_system();
      done.host[0] = *done.err;
      host_flag_set(done.host + 1, done.seq);
    }
  }
}

}  // namespace pihm

// ---------------------------------------------------------------------------
// launch helpers used by the host side
// ---------------------------------------------------------------------------
namespace pihm {

static inline unsigned blocks_for(long long n, int threads) {
  return (unsigned)((n + threads - 1) / threads);
}

// Take two events from the profiler's pool (grown on demand).
static bool prof_begin(Profiler *p, int kernel, cudaStream_t st) {
  if (!p) return false;
  if (p->used + 2 > p->npool) {
    int n = p->npool ? 2 * p->npool : 256;
    cudaEvent_t *np_ = (cudaEvent_t *)realloc(p->pool, sizeof(cudaEvent_t) * n);
    if (!np_) return false;
    p->pool = np_;
    for (int k = p->npool; k < n; k++) cudaEventCreate(&p->pool[k]);
    p->npool = n;
  }
  if (p->nrec + 1 > p->cap) {
    int n = p->cap ? 2 * p->cap : 128;
    Profiler::Rec *nr_ = (Profiler::Rec *)realloc(p->recs, sizeof(Profiler::Rec) * n);
    if (!nr_) return false;
    p->recs = nr_;
    p->cap = n;
  }
  Profiler::Rec &r = p->recs[p->nrec++];
  r.kernel = kernel;
  r.a = p->pool[p->used++];
  r.b = p->pool[p->used++];
  cudaEventRecord(r.a, st);
  return true;
}
static void prof_end(Profiler *p, bool on, cudaStream_t st) {
  if (on) cudaEventRecord(p->recs[p->nrec - 1].b, st);
}

// k_rhs_fused at 128 registers (2 x 256 threads per SM: the powers of a
// column overlap) and at 64 (4 x 256: twice as many items at once).
static const void *fused_kernel(int dense, bool from_ref) {
  if (dense) return from_ref ? (const void *)k_rhs_fused<true, 4> : (const void *)k_rhs_fused<false, 4>;
  return from_ref ? (const void *)k_rhs_fused<true, 2> : (const void *)k_rhs_fused<false, 2>;
}

// k_rhs_fused's resident blocks per launch, for 32, 64, 128 and 256 threads.
cudaError_t fused_plan(FusedPlan *f) {
  int dev = 0, sms = 0, coop = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  for (int d = 0; d < 2; d++)
    for (int k = 0; k < FusedPlan::kSizes && e == cudaSuccess; k++) {
      int a = 0, b = 0;
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, fused_kernel(d, false), 32 << k, 0);
      if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, fused_kernel(d, true), 32 << k, 0);
      f->blocks[d][k] = coop ? sms * std::min(a, b) : 0;
    }
  f->sms = sms;
  return e;
}

// How k_rhs_fused would run this evaluation: blocks as small as leave every
// SM a few warps, so that a small mesh spreads over the chip (an SM takes an
// FP64 warp instruction every 20 clocks), one item a thread.  False when the
// items are more than can be resident together: the blocks of one kind would
// then take turns while the others wait, and the separate kernels are faster.
struct FusedLaunch {
  FusedGrid g;
  int dense, threads;
};
static bool fused_fits(const DevMesh &m, const FusedPlan &f, bool from_ref, FusedLaunch *l) {
  const long long elems = from_ref ? m.ne + 2LL * m.nr : m.ne_run;
  const long long all = elems + m.nedge_run + (long long)kRivParts * m.nr_run + m.ne_run;
  if (!m.bar || m.ne_run <= 0 || all > 2048LL * f.sms) return false;
  int k = 0;
  while (k + 1 < FusedPlan::kSizes && all > (32LL << k) * f.sms) k++;
  l->threads = 32 << k;
  l->g = FusedGrid{(int)blocks_for(elems, l->threads), (int)blocks_for(m.nedge_run, l->threads),
                   kRivParts * (int)blocks_for(m.nr_run, l->threads), (int)blocks_for(m.ne_run, l->threads)};
  const int want = l->g.elem + l->g.edge + l->g.river + l->g.col;
  l->dense = want > f.blocks[0][k];
  return want <= f.blocks[l->dense][k];
}
static cudaError_t launch_fused(const DevMesh &m, FusedLaunch &l, const double *y, double *ydot, cudaStream_t st,
                                const double *y_ref, const int32_t *iperm) {
  double *y_int = const_cast<double *>(y);  // y_ref: the internal-order buffer the kernel fills
  void *args[] = {(void *)&m, (void *)&y, &ydot, (void *)&y_ref, &y_int, (void *)&iperm, &l.g};
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(l.g.elem + l.g.edge + l.g.river + l.g.col);
  cfg.blockDim = dim3(l.threads);
  cfg.stream = st;
  cudaLaunchAttribute at[2]{};
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  return launched(cudaLaunchKernelExC(&cfg, fused_kernel(l.dense, y_ref != nullptr), args));
}

template <class... P, class... A>
static cudaError_t launch_after(void (*kernel)(P...), dim3 grid, int block, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)block);
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return launched(cudaLaunchKernelEx(&cfg, kernel, P(args)...));
}

cudaError_t launch_rhs(const DevMesh &m, const double *y, double *ydot, cudaStream_t st,
                       long long *launches, Profiler *prof, const FusedPlan *fused, const double *y_ref,
                       const int32_t *iperm) {
  bool on;
  // a small mesh in one launch (per-kernel timing keeps the separate kernels):
  // one evaluation of 1,000 / 20,000 / 40,000 elements takes 16 / 21 / 29 us
  // (the five launches 43 for 60,000; as seven plain launches on two streams
  // the same meshes took 41 / 46 / 54)
  FusedLaunch fl;
  if (fused && !prof && fused_fits(m, *fused, y_ref != nullptr, &fl)) {
    ++*launches;
    return launch_fused(m, fl, y, ydot, st, y_ref, iperm);
  }
  // The river work rides in the element kernels' grids, ahead of the
  // elements: geometry with k_elem_prep, fluxes with k_elem_grad, rows with
  // k_bank_rows.  Per-kernel timing, and an arena without elements, keep
  // them apart.  Against river kernels on a second stream, its two events and
  // plain launches, with k_bank_rows's 10 us of latency at the end: 60,000
  // elements 55 -> 43 us, 200,000 103 -> 86, 400,000 171 -> 146, 1,000,000
  // 345 -> 322.
  const bool with = !prof && m.ne_run > 0 && m.nr_run > 0;
  const bool from_ref = y_ref != nullptr;
  const unsigned rows = m.nr_run > 0 ? blocks_for(m.nr_run, 128) : 0;
  const unsigned parts = m.nr_run > 0 ? kRivParts * ((m.nr_run + 31u) & ~31u) : 0;
  cudaError_t err = cudaSuccess;
  const auto after = [&](auto kernel, unsigned grid, int block, auto... args) {
    if (err == cudaSuccess) err = launch_after(kernel, dim3(grid), block, st, args...);
    ++*launches;
  };
  if (m.ne_run > 0) {
    on = prof_begin(prof, K_PREP, st);
    const unsigned geom = with ? blocks_for(m.nr_run, kPrepBlock) : 0;
    if (from_ref)  // y is the internal-order buffer the kernel fills
      after(k_elem_prep<true>, geom + blocks_for((long long)m.ne + 2LL * m.nr, kPrepBlock), kPrepBlock, m,
            (const double *)nullptr, y_ref, const_cast<double *>(y), iperm, (int)geom);
    else
      after(k_elem_prep<false>, geom + blocks_for(m.ne_run, kPrepBlock), kPrepBlock, m, y, (const double *)nullptr,
            (double *)nullptr, (const int32_t *)nullptr, (int)geom);
    prof_end(prof, on, st);
    const bool grad = m.surf_mode == kDiffWave;
    if (grad || with) {
      on = prof_begin(prof, K_GRAD, st);
      const unsigned river = with ? blocks_for(parts, 256) : 0;
      after(k_elem_grad, river + (grad ? blocks_for(m.ne_run, 256) : 0), 256, m, y, (int)river, from_ref);
      prof_end(prof, on, st);
    }
    if (m.nedge_run > 0) {
      on = prof_begin(prof, K_EDGE, st);
      after(k_edge, blocks_for(m.nedge_run, kEdgeBlock), kEdgeBlock, m, y);
      prof_end(prof, on, st);
    }
    on = prof_begin(prof, K_MAIN, st);
    switch (m.main_shape) {
      case 1: after(k_elem_main<256, 4>, blocks_for(m.ne_run, 256), 256, m, y, ydot, from_ref); break;
      case 2: after(k_elem_main<128, 8>, blocks_for(m.ne_run, 128), 128, m, y, ydot, from_ref); break;
      default: after(k_elem_main<512, 2>, blocks_for(m.ne_run, 512), 512, m, y, ydot, from_ref); break;
    }
    prof_end(prof, on, st);
  }
  if (!with && m.nr_run > 0) {
    on = prof_begin(prof, K_RIVER, st);
    k_riv_geom<<<rows, 128, 0, st>>>(m, y);
    k_river<<<blocks_for(parts, 128), 128, 0, st>>>(m, y);
    k_river_rows<<<rows, 128, 0, st>>>(m, ydot);
    prof_end(prof, on, st);
    *launches += 3;
  }
  const unsigned late = with ? rows : 0;
  if (late > 0 || m.nbank_run > 0) {
    on = prof_begin(prof, K_FINISH, st);
    after(k_bank_rows, late + (m.nbank_run > 0 ? blocks_for(m.nbank_run, 128) : 0), 128, m, ydot, (int)late);
    prof_end(prof, on, st);
  }
  const cudaError_t plain = cudaGetLastError();
  return err == cudaSuccess ? plain : err;
}

cudaError_t launch_permute(const double *src, double *dst, const int32_t *perm, int ne, int nr,
                           int to_internal, cudaStream_t st) {
  if (ne + 2LL * nr == 0) return cudaSuccess;
  return launch_after(k_permute, dim3(blocks_for(ne + 2LL * nr, 256), 3), 256, st, src, dst, perm, ne, nr, to_internal);
}

cudaError_t launch_permute_ref(const double *src, double *dst, const int32_t *iperm, int ne, int nr,
                               int to_internal, const StatusOut &done, cudaStream_t st) {
  if (ne + 2LL * nr == 0) return cudaSuccess;
  return launch_after(k_permute_ref, dim3(blocks_for(ne + 2LL * nr, 256), 3), 256, st, src, dst, iperm, ne, nr, to_internal, done);
}

}  // namespace pihm
