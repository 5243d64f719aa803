// The Noah land-surface model of Flux-PIHM on the device (include/pihm_noah.h).
//
// One thread per element and kernel:
//   k_noah_step   Noah() over a land-surface step (noah_phys.cuh: CalHum,
//                 FrozRain, net radiation, SFlx with its snowpack,
//                 frozen-soil, soil-heat and canopy physics)
//   k_noah_post   after a model step: Summary's _NOAH_ part (MassBalance's
//                 infiltration and subsurface runoff, src/update.c:100-165;
//                 runoff2, FindWaterTable, CalcLatFlx, src/update.c:34-41)
//                 and NoahHydrol (FindWaterTable, the moisture clamps, SmFlx,
//                 src/noah/noah.c:57-97)
// and both end with what the Flux-PIHM right-hand side reads (write_inputs;
// k_noah_inputs after a state is set): GwTransp's layer sum
// (noah/lsm_func.c:163-185) and whether the water table lies within the root
// zone, Infil's top-layer saturation (src/vert_flow.c:94-98), the frozen-soil
// factor, and the right-hand side's edir, ett and pcpdrp planes.
// Every plane is in the context's internal element order; per-layer planes
// are [layer][ne].  The state never leaves the device between steps.
#include <cmath>
#include <cstring>
#include <vector>

#include "noah_phys.cuh"
#include "pihm_internal.h"
#include "pihm_noah.h"

namespace pihm {

// scalar per-element planes
enum NoahScalar {
  // parameters
  NS_SMCMAX = 0, NS_SMCMIN, NS_SMCREF, NS_SMCWLT, NS_SMCDRY, NS_QUARTZ, NS_CSOIL, NS_ALPHA, NS_BETA, NS_KSATV,
  NS_POROSITY, NS_DEPTH, NS_AREA, NS_SHDFAC, NS_CMCFACTR, NS_LAIMAX, NS_LAIMIN, NS_EMISSMAX, NS_EMISSMIN,
  NS_ALBEDOMAX, NS_ALBEDOMIN, NS_Z0MAX, NS_Z0MIN, NS_SNUP, NS_CFACTR, NS_RGL, NS_RSMIN, NS_RSMAX, NS_TOPT, NS_HS,
  NS_SBETA, NS_SALP, NS_FRZX, NS_FXEXP, NS_CZIL, NS_LVCOEF, NS_ZBOT, NS_TBOT, NS_ZLVL, NS_ZLVL_WIND, NS_SNOALB,
  // forcing
  NS_PRCP, NS_SFCTMP, NS_RH, NS_SFCSPD, NS_SOLDN, NS_LONGWAVE, NS_SFCPRS, NS_LAI,
  // carried state
  NS_T1, NS_CMC, NS_SNEQV, NS_SNOWH, NS_SNDENS, NS_CH, NS_CM, NS_SNOTIME1, NS_ALBEDO, NS_EMISSI, NS_Q1, NS_RIBB,
  NS_FCR,
  // outputs
  NS_EDIR, NS_EC, NS_ETT, NS_ESNOW, NS_ETP, NS_DRIP, NS_PCPDRP, NS_SNOMLT, NS_SSOIL, NS_SHEAT, NS_RUNOFF2,
  NS_RUNOFF3, NS_INFIL, NS_SNCOVR, NS_BETA_S, NS_ETA, NS_SOILM,
  // kept from step to step like the reference's wf.etns, which SnoPac's dew
  // branch leaves unchanged and SFlx then reads
  NS_ETNS,
  // the previous model step's groundwater and unsaturated storage (ws0)
  NS_GW0, NS_UNSAT0,
  NS_COUNT
};
enum NoahLayer { NL_SLDPTH = 0, NL_ZSOIL, NL_RTDIS, NL_SMC, NL_SH2O, NL_STC, NL_ET, NL_RUNOFF2_LYR, NL_SMFLXV, NL_COUNT };
enum NoahInt { NI_NSOIL = 0, NI_NROOT, NI_ISURBAN, NI_NWTBL, NI_COUNT };

struct NoahPlanes {
  double *s[NS_COUNT];
  double *l[NL_COUNT];
  int32_t *i[NI_COUNT];
  int32_t *order;   // [ne] elements grouped by the branches Noah() will take (k_noah_classify)
  int32_t *cls;     // [2 * kNoahClasses] class sizes, then cursors
  int ne;
};

namespace {

using noah::Real;
constexpr int L = noah::kMaxLayers;

// What a land-surface step reads of a column.
template <class Col>
__device__ void load_col(const NoahPlanes &P, int i, Col &c) {
  const int ne = P.ne;
  c.nsoil = P.i[NI_NSOIL][i];
  c.nroot = P.i[NI_NROOT][i];
  c.isurban = P.i[NI_ISURBAN][i];
  c.nwtbl = P.i[NI_NWTBL][i];
#pragma unroll
  for (int k = 0; k < Col::L; k++)
    if (k < c.nsoil) {
      c.sldpth[k] = P.l[NL_SLDPTH][k * ne + i];
      c.zsoil[k] = P.l[NL_ZSOIL][k * ne + i];
      c.rtdis[k] = P.l[NL_RTDIS][k * ne + i];
      c.smc[k] = P.l[NL_SMC][k * ne + i];
      c.sh2o[k] = P.l[NL_SH2O][k * ne + i];
      c.stc[k] = P.l[NL_STC][k * ne + i];
      c.et[k] = P.l[NL_ET][k * ne + i];
    }
  const double *const *s = P.s;
  c.smcmax = s[NS_SMCMAX][i]; c.smcmin = s[NS_SMCMIN][i]; c.smcref = s[NS_SMCREF][i];
  c.smcwlt = s[NS_SMCWLT][i]; c.smcdry = s[NS_SMCDRY][i]; c.quartz = s[NS_QUARTZ][i];
  c.csoil = s[NS_CSOIL][i]; c.alpha = s[NS_ALPHA][i]; c.beta = s[NS_BETA][i]; c.ksatv = s[NS_KSATV][i];
  c.porosity = s[NS_POROSITY][i]; c.depth = s[NS_DEPTH][i]; c.area = s[NS_AREA][i];
  c.shdfac = s[NS_SHDFAC][i]; c.cmcfactr = s[NS_CMCFACTR][i]; c.laimax = s[NS_LAIMAX][i];
  c.laimin = s[NS_LAIMIN][i]; c.emissmax = s[NS_EMISSMAX][i]; c.emissmin = s[NS_EMISSMIN][i];
  c.albedomax = s[NS_ALBEDOMAX][i]; c.albedomin = s[NS_ALBEDOMIN][i]; c.z0max = s[NS_Z0MAX][i];
  c.z0min = s[NS_Z0MIN][i]; c.snup = s[NS_SNUP][i]; c.cfactr = s[NS_CFACTR][i]; c.rgl = s[NS_RGL][i];
  c.rsmin = s[NS_RSMIN][i]; c.rsmax = s[NS_RSMAX][i]; c.topt = s[NS_TOPT][i]; c.hs = s[NS_HS][i];
  c.sbeta = s[NS_SBETA][i]; c.salp = s[NS_SALP][i]; c.frzx = s[NS_FRZX][i]; c.fxexp = s[NS_FXEXP][i];
  c.czil = s[NS_CZIL][i]; c.lvcoef = s[NS_LVCOEF][i]; c.zbot = s[NS_ZBOT][i]; c.tbot = s[NS_TBOT][i];
  c.zlvl = s[NS_ZLVL][i]; c.zlvl_wind = s[NS_ZLVL_WIND][i]; c.snoalb = s[NS_SNOALB][i];
  c.prcp = s[NS_PRCP][i]; c.sfctmp = s[NS_SFCTMP][i]; c.rh = s[NS_RH][i]; c.sfcspd = s[NS_SFCSPD][i];
  c.soldn = s[NS_SOLDN][i]; c.longwave = s[NS_LONGWAVE][i]; c.sfcprs = s[NS_SFCPRS][i];
  c.proj_lai = s[NS_LAI][i];
  c.t1 = s[NS_T1][i]; c.cmc = s[NS_CMC][i]; c.sneqv = s[NS_SNEQV][i]; c.snowh = s[NS_SNOWH][i];
  c.sndens = s[NS_SNDENS][i]; c.ch = s[NS_CH][i]; c.cm = s[NS_CM][i]; c.snotime1 = s[NS_SNOTIME1][i];
  c.albedo = s[NS_ALBEDO][i]; c.emissi = s[NS_EMISSI][i]; c.q1 = s[NS_Q1][i]; c.ribb = s[NS_RIBB][i];
  c.fcr = s[NS_FCR][i];
  c.edir = s[NS_EDIR][i]; c.ec = s[NS_EC][i]; c.ett = s[NS_ETT][i]; c.esnow = s[NS_ESNOW][i];
  c.etp = s[NS_ETP][i]; c.drip = s[NS_DRIP][i]; c.pcpdrp = s[NS_PCPDRP][i]; c.snomlt = s[NS_SNOMLT][i];
  c.ssoil = s[NS_SSOIL][i]; c.sheat = s[NS_SHEAT][i]; c.sncovr = s[NS_SNCOVR][i];
  c.beta_s = s[NS_BETA_S][i]; c.eta = s[NS_ETA][i]; c.soilm = s[NS_SOILM][i];
  c.etns = s[NS_ETNS][i];
}

// What a step changes: the state, the outputs and -- for urban land, where
// SFlx overrides them for good (src/noah/noah.c:201-212) -- the parameters.
template <class Col>
__device__ void store_col(const NoahPlanes &P, int i, const Col &c) {
  const int ne = P.ne;
#pragma unroll
  for (int k = 0; k < Col::L; k++) {
    if (k >= c.nsoil) break;
    P.l[NL_SMC][k * ne + i] = c.smc[k].v;
    P.l[NL_SH2O][k * ne + i] = c.sh2o[k].v;
    P.l[NL_STC][k * ne + i] = c.stc[k].v;
    P.l[NL_ET][k * ne + i] = c.et[k].v;
  }
  double *const *s = P.s;
  if (c.isurban) {
    s[NS_SHDFAC][i] = c.shdfac.v; s[NS_RSMIN][i] = c.rsmin.v; s[NS_SMCMAX][i] = c.smcmax.v;
    s[NS_SMCMIN][i] = c.smcmin.v; s[NS_SMCREF][i] = c.smcref.v; s[NS_SMCWLT][i] = c.smcwlt.v;
    s[NS_SMCDRY][i] = c.smcdry.v;
  }
  s[NS_T1][i] = c.t1.v; s[NS_CMC][i] = c.cmc.v; s[NS_SNEQV][i] = c.sneqv.v; s[NS_SNOWH][i] = c.snowh.v;
  s[NS_SNDENS][i] = c.sndens.v; s[NS_CH][i] = c.ch.v; s[NS_CM][i] = c.cm.v; s[NS_SNOTIME1][i] = c.snotime1.v;
  s[NS_ALBEDO][i] = c.albedo.v; s[NS_EMISSI][i] = c.emissi.v; s[NS_Q1][i] = c.q1.v;
  s[NS_EDIR][i] = c.edir.v; s[NS_EC][i] = c.ec.v; s[NS_ETT][i] = c.ett.v; s[NS_ESNOW][i] = c.esnow.v;
  s[NS_ETP][i] = c.etp.v; s[NS_DRIP][i] = c.drip.v; s[NS_PCPDRP][i] = c.pcpdrp.v; s[NS_SNOMLT][i] = c.snomlt.v;
  s[NS_SSOIL][i] = c.ssoil.v; s[NS_SHEAT][i] = c.sheat.v; s[NS_SNCOVR][i] = c.sncovr.v;
  s[NS_BETA_S][i] = c.beta_s.v; s[NS_ETA][i] = c.eta.v; s[NS_SOILM][i] = c.soilm.v;
  s[NS_ETNS][i] = c.etns.v;
}

// The Flux-PIHM right-hand side's inputs from a column's state and outputs.
template <class Col>
__device__ __forceinline__ void write_inputs(const NoahTargets &o, int i, const Col &c) {
  Real g = 0.0;
  if (c.nwtbl <= c.nroot)
    for (int j = (c.nwtbl <= 0 ? 0 : c.nwtbl - 1); j < c.nroot; j++) g += c.et[j];
  o.etgw[i] = g.v;
  o.wtin[i] = c.nwtbl <= c.nroot;
  o.satn[i] = ((c.sh2o[0] - c.smcmin) / (c.smcmax - c.smcmin)).v;
  o.fcr[i] = c.fcr.v;
  o.edir[i] = c.edir.v;
  o.ett[i] = c.ett.v;
  o.pcpdrp[i] = c.pcpdrp.v;
}

constexpr int kNoahBlock = 128;
constexpr int kNoahClasses = 32;

// The branch class of an element's next Noah() step: whether it will run the
// snowpack path (snow on the ground, or precipitation that may fall as snow
// or freezing rain), whether the surface layer is unstable (SfcDifOff's
// logarithms and arctangents), how many layers hold ice or frost (each runs
// FrH2O's iterations, up to 7 told apart).  Noah() is one thread per element
// and an SM takes an FP64 warp instruction every 20 clocks, so a warp whose
// lanes take different paths runs each path for all of them; grouping elements
// by class keeps warps on one path.  Only the order of work changes: every
// element's arithmetic, and so every result, is the same.
__device__ __forceinline__ int noah_class(const NoahPlanes &P, int i) {
  const double tf = 273.15;
  const double sfctmp = P.s[NS_SFCTMP][i], t1 = P.s[NS_T1][i];
  const bool snow = P.s[NS_SNEQV][i] > 0.0 || (P.s[NS_PRCP][i] > 0.0 && sfctmp <= tf + 1.0);
  const int nsoil = P.i[NI_NSOIL][i];
  int frozen = t1 < tf;
  for (int k = 0; k < nsoil; k++)
    frozen += P.l[NL_STC][k * P.ne + i] < tf || P.l[NL_SMC][k * P.ne + i] > P.l[NL_SH2O][k * P.ne + i];
  const bool unstable = t1 > sfctmp + 0.0098 * P.s[NS_ZLVL][i];
  return (frozen < 7 ? frozen : 7) * 4 + (snow ? 2 : 0) + (unstable ? 1 : 0);
}

// class sizes (the caller zeroed cls): counted per block in shared
// memory, one global addition per class and block (one per element onto eight
// addresses took 60 us for 200,000 elements)
__global__ void __launch_bounds__(256) k_noah_count(NoahPlanes P) {
  __shared__ int n[kNoahClasses];
  if (threadIdx.x < kNoahClasses) n[threadIdx.x] = 0;
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int c = i < P.ne ? noah_class(P, i) : kNoahClasses;
  const unsigned mask = __match_any_sync(0xffffffffu, c);
  if (c < kNoahClasses && (int)(threadIdx.x & 31) == __ffs(mask) - 1) atomicAdd(&n[c], __popc(mask));
  __syncthreads();
  if (threadIdx.x < kNoahClasses && n[threadIdx.x]) atomicAdd(&P.cls[threadIdx.x], n[threadIdx.x]);
}

// each element's place: its class's start (the sizes of the classes after it,
// so that the longest columns, snow and frost, start first) plus a cursor;
// lanes of a warp in one class take consecutive places
__global__ void __launch_bounds__(256) k_noah_place(NoahPlanes P) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool in = i < P.ne;
  const int c = in ? noah_class(P, i) : kNoahClasses;
  const unsigned mask = __match_any_sync(0xffffffffu, c);
  if (!in) return;
  const int lead = __ffs(mask) - 1, lane = threadIdx.x & 31;
  int base = 0;
  if (lane == lead) base = atomicAdd(&P.cls[kNoahClasses + c], __popc(mask));
  base = __shfl_sync(mask, base, lead);
  int start = 0;
  for (int k = kNoahClasses - 1; k > c; k--) start += P.cls[k];
  P.order[start + base + __popc(mask & ((1u << lane) - 1u))] = i;
}

// kLayers: the most layers any column has (4, the usual Noah column, or 11):
// a column's layer arrays stand in local memory, 1 KB instead of 2.4.
template <int kLayers>
__global__ void __launch_bounds__(kNoahBlock, 4) k_noah_step(NoahPlanes P, NoahTargets o, double dt,
                                                             unsigned int *err) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= P.ne) return;
  const int i = P.order[t];
  noah::Layers<kLayers> layers;
  noah::ColT<kLayers> c(layers);
  load_col(P, i, c);
  noah::noah_step(c, Real(dt));
  // the reference exits when the snow density exceeds one (SFlx) or a
  // state turns NaN; here the context's error word records it
  if (c.sneqv > 1.0e-7 && !(c.sndens <= 1.0)) atomicOr(err, 1u);
  if (c.t1 != c.t1 || c.edir != c.edir || c.ett != c.ett) atomicOr(err, 1u);
  store_col(P, i, c);
  write_inputs(o, i, c);
}

// The branches a column takes in the post-step: saturated (nothing but its
// moisture is set), without ice, or with ice, which takes the conductivity's
// powers twice.  A block's elements are ranked by them, as in Noah()'s order
// but within the block, so that its loads stay close together: 327 -> 308 us
// for 200,000 elements (by Noah()'s own order 324; over blocks of 256 or 512
// threads 328 and 346: their last warps hold the SM alone).
constexpr int kPostClasses = 4;  // the last: past the end
__device__ __forceinline__ int post_class(const NoahPlanes &P, const double *y, int i) {
  const int nsoil = P.i[NI_NSOIL][i];
  double depth = 0.0;
  bool ice = false;
  for (int k = 0; k < nsoil; k++) {
    depth += P.l[NL_SLDPTH][k * P.ne + i];
    ice = ice || P.l[NL_SMC][k * P.ne + i] > P.l[NL_SH2O][k * P.ne + i];
  }
  return y[2 * P.ne + i] > depth ? 0 : (ice ? 1 : 2);
}

// y: the model state after the step (internal order); first: no previous
// state yet, ws0 is taken from y.  Only what the soil moisture needs of a
// column moves: 23 scalars and 7 layer planes in, 9 and 4 out, of the 85 and 9
// of a land-surface step.  200,000 elements: 0.33 ms instead of 0.72, the FP64
// pipe 62 % busy with the layers' additions and products.
template <int kLayers>
__global__ void __launch_bounds__(kNoahBlock, 4) k_noah_post(NoahPlanes P, NoahTargets o, const double *y, double dt,
                                                             int first) {
  __shared__ int s_n[kPostClasses][kNoahBlock / 32];
  __shared__ unsigned short s_order[kNoahBlock];
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  {
    const int cls = i < P.ne ? post_class(P, y, i) : kPostClasses - 1;
    const unsigned peers = __match_any_sync(0xffffffffu, cls);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int k = threadIdx.x; k < kPostClasses * (kNoahBlock / 32); k += kNoahBlock) (&s_n[0][0])[k] = 0;
    __syncthreads();
    if (lane == __ffs(peers) - 1) s_n[cls][warp] = __popc(peers);
    __syncthreads();
    int at = __popc(peers & ((1u << lane) - 1u));
    for (int k = 0; k < kPostClasses; k++)
      for (int w = 0; w < kNoahBlock / 32; w++)
        if (k < cls || (k == cls && w < warp)) at += s_n[k][w];
    s_order[at] = (unsigned short)threadIdx.x;
    __syncthreads();
    i = blockIdx.x * blockDim.x + s_order[threadIdx.x];
  }
  if (i >= P.ne) return;
  const int ne = P.ne;
  double *const *s = P.s;
  noah::Layers<kLayers> layers;
  noah::ColT<kLayers> c(layers);
  c.nsoil = P.i[NI_NSOIL][i];
  c.nroot = P.i[NI_NROOT][i];
#pragma unroll
  for (int k = 0; k < kLayers; k++)
    if (k < c.nsoil) {
      c.sldpth[k] = P.l[NL_SLDPTH][k * ne + i];
      c.zsoil[k] = P.l[NL_ZSOIL][k * ne + i];
      c.smc[k] = P.l[NL_SMC][k * ne + i];
      c.sh2o[k] = P.l[NL_SH2O][k * ne + i];
      c.et[k] = P.l[NL_ET][k * ne + i];
      c.runoff2_lyr[k] = P.l[NL_RUNOFF2_LYR][k * ne + i];
    }
  c.smcmax = s[NS_SMCMAX][i]; c.smcmin = s[NS_SMCMIN][i]; c.alpha = s[NS_ALPHA][i]; c.beta = s[NS_BETA][i];
  c.ksatv = s[NS_KSATV][i]; c.porosity = s[NS_POROSITY][i]; c.depth = s[NS_DEPTH][i]; c.area = s[NS_AREA][i];
  c.frzx = s[NS_FRZX][i]; c.fcr = s[NS_FCR][i];
  c.edir = s[NS_EDIR][i]; c.ett = s[NS_ETT][i]; c.pcpdrp = s[NS_PCPDRP][i];
  // Summary, src/update.c:3-48: the element state from y, then MassBalance
  const Real unsat = y[ne + i], gw = y[2 * ne + i];
  const Real gw0 = first ? gw : Real(s[NS_GW0][i]);
  const Real unsat0 = first ? unsat : Real(s[NS_UNSAT0][i]);
  Real soilw0 = gw0 + unsat0;
  soilw0 = (soilw0 > c.depth) ? c.depth : soilw0;
  soilw0 = (soilw0 < 0.0) ? 0.0 : soilw0;
  Real soilw1 = gw + unsat;
  soilw1 = (soilw1 > c.depth) ? c.depth : soilw1;
  soilw1 = (soilw1 < 0.0) ? 0.0 : soilw1;
  Real subrunoff = 0.0;
  const int64_t ds = o.stride;
  for (int j = 0; j < 3; j++) subrunoff += Real(o.d_sub[j * ds + i]) / c.area;
  // the last evaluation's ET split: edir_unsat, edir_gw, ett_unsat, ett_gw
  c.infil = (soilw1 - soilw0) * c.porosity / dt + subrunoff + o.d_et[ds + i] + o.d_et[2 * ds + i] +
            o.d_et[3 * ds + i] + o.d_et[4 * ds + i];
  if (c.infil < 0.0) {
    subrunoff -= c.infil;
    c.infil = 0.0;
  }
  c.runoff2 = subrunoff;
  c.nwtbl = noah::find_water_table<kLayers>(c.sldpth, c.nsoil, gw, c.satdpth);
  noah::calc_lat_flx(c);
  s[NS_GW0][i] = gw.v;
  s[NS_UNSAT0][i] = unsat.v;
  // NoahHydrol
  noah::noah_hydrol(c, Real(dt));
#pragma unroll
  for (int k = 0; k < kLayers; k++) {
    if (k >= c.nsoil) break;
    P.l[NL_SMC][k * ne + i] = c.smc[k].v;
    P.l[NL_SH2O][k * ne + i] = c.sh2o[k].v;
    P.l[NL_RUNOFF2_LYR][k * ne + i] = c.runoff2_lyr[k].v;
  }
  P.i[NI_NWTBL][i] = c.nwtbl;
  s[NS_INFIL][i] = c.infil.v;
  s[NS_RUNOFF2][i] = c.runoff2.v;
  if (c.nwtbl != 0) {  // else SmFlx only saturated the column
#pragma unroll
    for (int k = 0; k < kLayers; k++) {
      if (k >= c.nsoil) break;
      P.l[NL_SMFLXV][k * ne + i] = c.smflxv[k].v;
    }
    s[NS_FCR][i] = c.fcr.v;
    s[NS_RUNOFF3][i] = c.runoff3.v;
  }
  write_inputs(o, i, c);
}

// ws0 from the state a run starts from
__global__ void __launch_bounds__(256) k_noah_begin(NoahPlanes P, const double *y) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= P.ne) return;
  P.s[NS_UNSAT0][i] = y[P.ne + i];
  P.s[NS_GW0][i] = y[2 * P.ne + i];
}

// The Flux-PIHM right-hand side's inputs from Noah's state and outputs.
__global__ void __launch_bounds__(256) k_noah_inputs(NoahPlanes P, NoahTargets o) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= P.ne) return;
  const int ne = P.ne;
  const int top = P.i[NI_NWTBL][i], nr = P.i[NI_NROOT][i];
  double g = 0.0;
  if (top <= nr)
    for (int j = (top <= 0 ? 0 : top - 1); j < nr; j++) g += P.l[NL_ET][j * ne + i];
  const double smcmin = P.s[NS_SMCMIN][i], smcmax = P.s[NS_SMCMAX][i];
  o.etgw[i] = g;
  o.wtin[i] = top <= nr;
  o.satn[i] = (P.l[NL_SH2O][i] - smcmin) / (smcmax - smcmin);
  o.fcr[i] = P.s[NS_FCR][i];
  o.edir[i] = P.s[NS_EDIR][i];
  o.ett[i] = P.s[NS_ETT][i];
  o.pcpdrp[i] = P.s[NS_PCPDRP][i];
}

template <class T>
size_t padded(size_t n) {
  return (n * sizeof(T) + 255) & ~size_t(255);
}

int cuda_rc(cudaError_t e) { return e == cudaSuccess ? PIHM_GPU_OK : PIHM_GPU_ERR_CUDA; }

// reference-order [ne][per] host values -> internal-order [per][ne] device planes
int upload(const int32_t *perm, int ne, const double *src, int per, double *const *dst, cudaStream_t st) {
  std::vector<double> h((size_t)ne);
  for (int k = 0; k < per; k++) {
    for (int i = 0; i < ne; i++) h[i] = src[(size_t)per * perm[i] + k];
    if (cudaMemcpyAsync(dst[k], h.data(), sizeof(double) * ne, cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
      return PIHM_GPU_ERR_CUDA;
  }
  return PIHM_GPU_OK;
}

int upload_layers(const int32_t *perm, int ne, const double *src, double *plane, cudaStream_t st) {
  double *dst[noah::kMaxLayers];
  for (int k = 0; k < noah::kMaxLayers; k++) dst[k] = plane + (size_t)k * ne;
  return upload(perm, ne, src, noah::kMaxLayers, dst, st);
}

int upload_int(const int32_t *perm, int ne, const int32_t *src, int32_t *dst) {
  std::vector<int32_t> h((size_t)ne);
  for (int i = 0; i < ne; i++) h[i] = src[perm[i]];
  return cuda_rc(cudaMemcpy(dst, h.data(), sizeof(int32_t) * ne, cudaMemcpyHostToDevice));
}

int upload_scalar(const int32_t *perm, int ne, const double *src, double *dst, cudaStream_t st) {
  return src ? upload(perm, ne, src, 1, &dst, st) : 0;
}

int launch_inputs(NoahInstance &n, cudaStream_t st, int64_t *launches) {
  k_noah_inputs<<<(n.ne + 255) / 256, 256, 0, st>>>(*n.P, n.tg);
  ++*launches;
  return cuda_rc(cudaGetLastError());
}

}  // namespace

int noah_set_state(NoahInstance &n, const pihm_noah_state *s, const int32_t *perm, cudaStream_t st) {
  if (!n.alloc || !s) return PIHM_GPU_ERR_ARG;
  NoahPlanes &P = *n.P;
  const int ne = n.ne;
  int rc = PIHM_GPU_OK;
  if (s->smc) rc = rc ?: upload_layers(perm, ne, s->smc, P.l[NL_SMC], st);
  if (s->sh2o) rc = rc ?: upload_layers(perm, ne, s->sh2o, P.l[NL_SH2O], st);
  if (s->stc) rc = rc ?: upload_layers(perm, ne, s->stc, P.l[NL_STC], st);
  const double *src[] = {s->t1, s->cmc, s->sneqv, s->snowh, s->sndens, s->ch, s->cm, s->snotime1,
                         s->albedo, s->emissi, s->q1, s->ribb, s->fcr};
  const int dst[] = {NS_T1, NS_CMC, NS_SNEQV, NS_SNOWH, NS_SNDENS, NS_CH, NS_CM, NS_SNOTIME1,
                     NS_ALBEDO, NS_EMISSI, NS_Q1, NS_RIBB, NS_FCR};
  for (int k = 0; k < 13; k++) rc = rc ?: upload_scalar(perm, ne, src[k], P.s[dst[k]], st);
  int64_t launches = 0;
  return rc ?: launch_inputs(n, st, &launches) ?: cuda_rc(cudaStreamSynchronize(st));
}

int noah_build(const pihm_noah_params *p, const pihm_noah_state *s, const int32_t *perm, int ne,
               const NoahTargets &tg, cudaStream_t st, NoahInstance *out) {
  if (!p || !s || !out || p->nelem != ne || !p->nsoil || !p->sldpth || !p->nroot || !p->rtdis) return PIHM_GPU_ERR_ARG;
  int layers = 0;
  for (int r = 0; r < ne; r++) {
    // HRT and SRT read the second layer: at least two
    if (p->nsoil[r] < 2 || p->nsoil[r] > noah::kMaxLayers || p->nroot[r] < 1 || p->nroot[r] > p->nsoil[r])
      return PIHM_GPU_ERR_ARG;
    if (p->nsoil[r] > layers) layers = p->nsoil[r];
  }
  const double *params[] = {p->smcmax, p->smcmin, p->smcref, p->smcwlt, p->smcdry, p->quartz, p->csoil,
                            p->alpha, p->beta, p->ksatv, p->porosity, p->depth, p->area, p->shdfac,
                            p->cmcfactr, p->laimax, p->laimin, p->emissmax, p->emissmin, p->albedomax,
                            p->albedomin, p->z0max, p->z0min, p->snup, p->cfactr, p->rgl, p->rsmin,
                            p->rsmax, p->topt, p->hs, p->sbeta, p->salp, p->frzx, p->fxexp, p->czil,
                            p->lvcoef, p->zbot, p->tbot, p->zlvl, p->zlvl_wind, p->snoalb};
  constexpr int kParams = NS_SNOALB + 1;
  static_assert(sizeof(params) / sizeof(params[0]) == kParams, "parameter list");
  for (const double *q : params)
    if (!q) return PIHM_GPU_ERR_ARG;
  if (!s->smc || !s->sh2o || !s->stc || !s->t1 || !s->cmc || !s->sneqv || !s->snowh || !s->sndens || !s->ch ||
      !s->cm || !s->snotime1 || !s->albedo || !s->emissi || !s->q1 || !s->ribb || !s->fcr)
    return PIHM_GPU_ERR_ARG;
  const size_t NE = ne;
  const size_t bytes = NS_COUNT * padded<double>(NE) + NL_COUNT * padded<double>(noah::kMaxLayers * NE) +
                       NI_COUNT * padded<int32_t>(NE) + padded<int32_t>(NE) + padded<int32_t>(2 * kNoahClasses);
  NoahInstance n;
  if (cudaMalloc(&n.alloc, bytes) != cudaSuccess) return PIHM_GPU_ERR_NOMEM;
  n.P = new NoahPlanes();
  n.tg = tg;
  n.ne = ne;
  n.first = 1;
  n.layers = layers;
  if (cudaMemset(n.alloc, 0, bytes) != cudaSuccess) {
    noah_release(n);
    return PIHM_GPU_ERR_CUDA;
  }
  NoahPlanes &P = *n.P;
  P.ne = ne;
  char *cur = (char *)n.alloc;
  for (int k = 0; k < NS_COUNT; k++) {
    P.s[k] = (double *)cur;
    cur += padded<double>(NE);
  }
  for (int k = 0; k < NL_COUNT; k++) {
    P.l[k] = (double *)cur;
    cur += padded<double>(noah::kMaxLayers * NE);
  }
  for (int k = 0; k < NI_COUNT; k++) {
    P.i[k] = (int32_t *)cur;
    cur += padded<int32_t>(NE);
  }
  P.order = (int32_t *)cur;
  cur += padded<int32_t>(NE);
  P.cls = (int32_t *)cur;
  int rc = PIHM_GPU_OK;
  for (int k = 0; k < kParams && !rc; k++) rc = upload_scalar(perm, ne, params[k], P.s[k], st);
  // layer depths below the surface (DefSldpth, noah/lsm_func.c:152-156)
  std::vector<double> zsoil((size_t)noah::kMaxLayers * ne, 0.0);
  for (int r = 0; r < ne; r++) {
    const double *sl = p->sldpth + (size_t)noah::kMaxLayers * r;
    double *z = zsoil.data() + (size_t)noah::kMaxLayers * r;
    z[0] = -sl[0];
    for (int k = 1; k < p->nsoil[r]; k++) z[k] = -sl[k] + z[k - 1];
  }
  rc = rc ?: upload_layers(perm, ne, p->sldpth, P.l[NL_SLDPTH], st);
  rc = rc ?: upload_layers(perm, ne, zsoil.data(), P.l[NL_ZSOIL], st);
  rc = rc ?: upload_layers(perm, ne, p->rtdis, P.l[NL_RTDIS], st);
  rc = rc ?: upload_int(perm, ne, p->nsoil, P.i[NI_NSOIL]);
  rc = rc ?: upload_int(perm, ne, p->nroot, P.i[NI_NROOT]);
  if (p->isurban) rc = rc ?: upload_int(perm, ne, p->isurban, P.i[NI_ISURBAN]);
  // the water-table layer before the first post-step: below the column
  std::vector<int32_t> nw((size_t)ne);
  for (int r = 0; r < ne; r++) nw[r] = p->nsoil[r];
  rc = rc ?: upload_int(perm, ne, nw.data(), P.i[NI_NWTBL]);
  rc = rc ?: noah_set_state(n, s, perm, st);
  if (rc) {
    noah_release(n);
    return rc;
  }
  *out = n;
  return PIHM_GPU_OK;
}

int noah_set_forcing(NoahInstance &n, const pihm_noah_forcing *f, const int32_t *perm, cudaStream_t st) {
  if (!n.alloc || !f || !f->prcp || !f->sfctmp || !f->rh || !f->sfcspd || !f->soldn || !f->longwave ||
      !f->sfcprs || !f->lai)
    return PIHM_GPU_ERR_ARG;
  NoahPlanes &P = *n.P;
  const double *src[] = {f->prcp, f->sfctmp, f->rh, f->sfcspd, f->soldn, f->longwave, f->sfcprs, f->lai};
  int rc = PIHM_GPU_OK;
  for (int k = 0; k < 8 && !rc; k++) rc = upload_scalar(perm, n.ne, src[k], P.s[NS_PRCP + k], st);
  return rc;
}

int noah_launch_step(NoahInstance &n, double dt, unsigned int *err, cudaStream_t st, int64_t *launches) {
  if (!n.alloc || !(dt > 0.0)) return PIHM_GPU_ERR_ARG;
  if (n.ne == 0) return PIHM_GPU_OK;
  if (cudaMemsetAsync(n.P->cls, 0, sizeof(int32_t) * 2 * kNoahClasses, st) != cudaSuccess) return PIHM_GPU_ERR_CUDA;
  k_noah_count<<<(n.ne + 255) / 256, 256, 0, st>>>(*n.P);
  k_noah_place<<<(n.ne + 255) / 256, 256, 0, st>>>(*n.P);
  const int blocks = (n.ne + kNoahBlock - 1) / kNoahBlock;
  if (n.layers <= 4) k_noah_step<4><<<blocks, kNoahBlock, 0, st>>>(*n.P, n.tg, dt, err);
  else k_noah_step<L><<<blocks, kNoahBlock, 0, st>>>(*n.P, n.tg, dt, err);
  *launches += 3;
  return cuda_rc(cudaGetLastError());
}

int noah_launch_begin(NoahInstance &n, const double *y0, cudaStream_t st, int64_t *launches) {
  if (!n.alloc || !y0) return PIHM_GPU_ERR_ARG;
  k_noah_begin<<<(n.ne + 255) / 256, 256, 0, st>>>(*n.P, y0);
  n.first = 0;
  ++*launches;
  return cuda_rc(cudaGetLastError());
}

int noah_launch_post(NoahInstance &n, const double *y, double dt, cudaStream_t st, int64_t *launches) {
  if (!n.alloc || !y || !(dt > 0.0)) return PIHM_GPU_ERR_ARG;
  const int blocks = (n.ne + kNoahBlock - 1) / kNoahBlock;
  if (n.layers <= 4) k_noah_post<4><<<blocks, kNoahBlock, 0, st>>>(*n.P, n.tg, y, dt, n.first);
  else k_noah_post<L><<<blocks, kNoahBlock, 0, st>>>(*n.P, n.tg, y, dt, n.first);
  n.first = 0;
  ++*launches;
  return cuda_rc(cudaGetLastError());
}

int noah_get(NoahInstance &n, int field, const int32_t *perm, cudaStream_t st, double *out) {
  if (!n.alloc || !out || field < 0 || field >= PIHM_NOAH_NFIELDS) return PIHM_GPU_ERR_ARG;
  const NoahPlanes &P = *n.P;
  const int ne = n.ne;
  if (cudaStreamSynchronize(st) != cudaSuccess) return PIHM_GPU_ERR_CUDA;
  static const int layer_of[] = {NL_SMC, NL_SH2O, NL_STC, NL_ET, NL_RUNOFF2_LYR, NL_SMFLXV};
  if (field < 6) {
    std::vector<double> h((size_t)noah::kMaxLayers * ne);
    if (cudaMemcpy(h.data(), P.l[layer_of[field]], sizeof(double) * h.size(), cudaMemcpyDeviceToHost) != cudaSuccess)
      return PIHM_GPU_ERR_CUDA;
    for (int k = 0; k < noah::kMaxLayers; k++)
      for (int i = 0; i < ne; i++) out[(size_t)noah::kMaxLayers * perm[i] + k] = h[(size_t)k * ne + i];
    return PIHM_GPU_OK;
  }
  static const int scalar_of[] = {NS_T1, NS_CMC, NS_SNEQV, NS_SNOWH, NS_SNDENS, NS_CH, NS_CM, NS_ALBEDO,
                                  NS_EMISSI, NS_Q1, NS_FCR, NS_EDIR, NS_EC, NS_ETT, NS_ESNOW, NS_ETP,
                                  NS_DRIP, NS_PCPDRP, NS_SNOMLT, NS_SSOIL, NS_SHEAT, NS_RUNOFF2, NS_RUNOFF3,
                                  NS_INFIL, -1, NS_SNOTIME1, NS_SNCOVR, NS_BETA_S, NS_ETA, NS_SOILM};
  const int idx = field - PIHM_NOAH_T1;
  if (field < PIHM_NOAH_T1 || idx >= (int)(sizeof(scalar_of) / sizeof(int))) return PIHM_GPU_ERR_ARG;
  std::vector<double> h((size_t)ne);
  if (scalar_of[idx] < 0) {  // nwtbl
    std::vector<int32_t> w((size_t)ne);
    if (cudaMemcpy(w.data(), P.i[NI_NWTBL], sizeof(int32_t) * ne, cudaMemcpyDeviceToHost) != cudaSuccess)
      return PIHM_GPU_ERR_CUDA;
    for (int i = 0; i < ne; i++) h[i] = w[i];
  } else if (cudaMemcpy(h.data(), P.s[scalar_of[idx]], sizeof(double) * ne, cudaMemcpyDeviceToHost) !=
             cudaSuccess) {
    return PIHM_GPU_ERR_CUDA;
  }
  for (int i = 0; i < ne; i++) out[perm[i]] = h[i];
  return PIHM_GPU_OK;
}

void noah_release(NoahInstance &n) {
  if (n.alloc) cudaFree(n.alloc);
  delete n.P;
  n = NoahInstance();
}

}  // namespace pihm

using namespace pihm;

extern "C" int pihm_gpu_noah_set_state(pihm_gpu_ctx *c, const pihm_noah_state *s) {
  if (!c || !c->noahlsm.alloc || !s) return PIHM_GPU_ERR_ARG;
  return noah_set_state(c->noahlsm, s, c->h_perm, c->stream);
}

extern "C" int pihm_gpu_noah_init(pihm_gpu_ctx *c, const pihm_noah_params *p, const pihm_noah_state *s) {
  if (!c || !p || !s || p->nelem != c->ne) return PIHM_GPU_ERR_ARG;
  const size_t NE = c->ne;
  // the right-hand side's Flux-PIHM input planes
  if (!c->d_noah) {
    const size_t nb = 3 * padded<double>(NE) + padded<int32_t>(NE);
    if (cudaMalloc(&c->d_noah, nb) != cudaSuccess) {
      c->d_noah = nullptr;
      return PIHM_GPU_ERR_NOMEM;
    }
    char *q = (char *)c->d_noah;
    c->m.noah_etgw = (double *)q; q += padded<double>(NE);
    c->m.noah_satn = (double *)q; q += padded<double>(NE);
    c->m.noah_fcr = (double *)q; q += padded<double>(NE);
    c->m.noah_wtin = (int32_t *)q;
  }
  NoahTargets tg{c->m.d_sub, c->m.d_et, (int64_t)c->ne, const_cast<double *>(c->m.noah_etgw),
                 const_cast<double *>(c->m.noah_satn), const_cast<double *>(c->m.noah_fcr),
                 const_cast<double *>(c->m.edir), const_cast<double *>(c->m.ett), const_cast<double *>(c->m.pcpdrp),
                 const_cast<int32_t *>(c->m.noah_wtin)};
  noah_release(c->noahlsm);
  const int rc = noah_build(p, s, c->h_perm, c->ne, tg, c->stream, &c->noahlsm);
  if (rc != PIHM_GPU_OK) return rc;
  c->m.noah = 1;
  c->diag = 1;  // MassBalance reads the last evaluation's fluxes
  return PIHM_GPU_OK;
}

extern "C" int pihm_gpu_noah_set_forcing(pihm_gpu_ctx *c, const pihm_noah_forcing *f) {
  if (!c || !c->noahlsm.alloc) return PIHM_GPU_ERR_ARG;
  return noah_set_forcing(c->noahlsm, f, c->h_perm, c->stream);
}

extern "C" int pihm_gpu_noah_step(pihm_gpu_ctx *c, double dt) {
  if (!c || !c->noahlsm.alloc) return PIHM_GPU_ERR_ARG;
  int64_t n = 0;
  const int rc = noah_launch_step(c->noahlsm, dt, c->m.err, c->stream, &n);
  c->launches += n;
  return rc;
}

extern "C" int pihm_gpu_noah_begin(pihm_gpu_ctx *c, const double *y0_dev) {
  if (!c || !c->noahlsm.alloc) return PIHM_GPU_ERR_ARG;
  int64_t n = 0;
  const int rc = noah_launch_begin(c->noahlsm, y0_dev, c->stream, &n);
  c->launches += n;
  return rc;
}

extern "C" int pihm_gpu_noah_post_step(pihm_gpu_ctx *c, const double *y_dev, double stepsize) {
  if (!c || !c->noahlsm.alloc) return PIHM_GPU_ERR_ARG;
  int64_t n = 0;
  const int rc = noah_launch_post(c->noahlsm, y_dev, stepsize, c->stream, &n);
  c->launches += n;
  return rc;
}

extern "C" int pihm_gpu_noah_get(pihm_gpu_ctx *c, int field, double *out) {
  if (!c || !c->noahlsm.alloc) return PIHM_GPU_ERR_ARG;
  return noah_get(c->noahlsm, field, c->h_perm, c->stream, out);
}
