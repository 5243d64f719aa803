"""Performance cases: the work a user of this library has it do, through its
public entry points, over the range of sizes that the tests, the benchmark and
the generator cover (1,000 to 1,000,000 elements in one watershed, batches of
small watersheds, vectors of 3,000 to 3,000,000 entries).

  rhs       the right-hand side on device-resident states (pihm_gpu_rhs)
  host      the same evaluation from host arrays (pihm_gpu_rhs_host), as a CPU
            integrator calls it in place of ODE()
  ensemble  independent states on several contexts of one mesh, each on a
            stream of its own
  vec       the N_Vector operations of one Newton / GMRES iteration
  land      the land-surface step at the start of a land-surface interval and
            the evaluation after it
  flux      Flux-PIHM's land-surface model over an interval: Noah, then model
            steps of one evaluation and the post-step update
  solve     the integrator over model steps on the plain path
  batch     watersheds of different sizes admitted, integrated together and
            read back

A case's watershed is the generator's (a user keeps one watershed and
evaluates many states on it); the states, the forcing and the vectors are
drawn from the seed.
"""
import ctypes
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "pihm-cuda_gb300"))

import pihm_gpu.land as LAND  # noqa: E402
import pihm_gpu.noah as NOAH  # noqa: E402
import pihm_gpu.nvector as NV  # noqa: E402
import pihm_gpu.watershed as W  # noqa: E402
import pihm_gpu.workloads as WL  # noqa: E402
from pihm_gpu.batch import Batch, limits_for  # noqa: E402
from pihm_gpu.capi import GpuRhs  # noqa: E402
from pihm_gpu.single import GpuWatershed  # noqa: E402
from pihm_gpu.solver import StepControl, run_steps  # noqa: E402

RELTOL, ABSTOL = 1e-4, 1e-5  # the benchmark's solver tolerances
LSM_STEP = 900.0             # the land-surface interval of the example deck (s)
LAND_START, LAND_HOURS = "2009-01-01 00:00", 48


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the 1,000-element configuration: one call of an integrator whose
        # every evaluation is latency
        dict(name="rhs_1k", kind="rhs", nelem=1000, mesh="grid", mode=2),
        # an unstructured mesh of an odd size under kinematic overland flow
        dict(name="rhs_kin_21k", kind="rhs", nelem=21483, mesh="scattered", mode=1),
        # the benchmark's headline: one evaluation of the 1M-element watershed
        dict(name="rhs_1m", kind="rhs", nelem=1_000_000, mesh="grid", mode=2),
        # the drop-in call of a CPU integrator at the Flux-PIHM mesh's size
        dict(name="host_200k", kind="host", nelem=200_000, mesh="grid"),
        # an ensemble of perturbed states of one watershed
        dict(name="ensemble_400k", kind="ensemble", nelem=400_000, mesh="grid", contexts=4, states=8),
        # a Newton / GMRES iteration's vector work, a small watershed and the
        # 1M-element one
        dict(name="vec_31k", kind="vec", n=31_337),
        dict(name="vec_3m", kind="vec", n=3_060_000),
        # a land-surface interval's start with station forcing
        dict(name="land_400k", kind="land", nelem=400_000, mesh="grid", stations=64, nlai=8),
        # the Flux-PIHM configuration: 200,000 elements, 4 Noah layers
        dict(name="flux_200k", kind="flux", nelem=200_000, mesh="grid", steps=6),
        # a small watershed solved alone: one model step of the integrator
        dict(name="solve_2k", kind="solve", nelem=2000, mesh="grid", steps=1),
        # many small watersheds at once, as calibration runs them
        dict(name="batch_24", kind="batch", systems=24, lo=2000, hi=20_000, steps=1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rhs", "rhs", "rhs", "host", "ensemble", "vec", "vec", "land", "flux", "solve", "batch"])
    mesh = rng.choice(["grid", "scattered"])
    if kind == "rhs":
        return dict(kind="rhs", nelem=_log_int(rng, 1000, 500_000), mesh=mesh, mode=rng.choice([1, 2, 2]))
    if kind == "host":
        return dict(kind="host", nelem=_log_int(rng, 1000, 200_000), mesh=mesh)
    if kind == "ensemble":
        return dict(kind="ensemble", nelem=_log_int(rng, 2000, 200_000), mesh=mesh, contexts=rng.choice([2, 3, 4]),
                    states=rng.choice([4, 6, 7]))
    if kind == "vec":
        return dict(kind="vec", n=_log_int(rng, 3000, 3_000_000))
    if kind == "land":
        return dict(kind="land", nelem=_log_int(rng, 1000, 300_000), mesh=mesh, stations=rng.randint(1, 64),
                    nlai=rng.randint(1, 8))
    if kind == "flux":
        return dict(kind="flux", nelem=_log_int(rng, 1000, 100_000), mesh=mesh, steps=rng.choice([4, 6]))
    if kind == "solve":
        return dict(kind="solve", nelem=_log_int(rng, 1000, 20_000), mesh=mesh, steps=1)
    return dict(kind="batch", systems=rng.randint(8, 20), lo=1000, hi=_log_int(rng, 4000, 20_000), steps=1)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=3)
def _mesh(nelem, mesh, mode=2):
    ws = W.generate(nelem, WL.river_count(nelem), seed=0, mesh=mesh)
    ws.surf_mode = mode
    return ws


def _rng(seed, what):
    return np.random.default_rng((seed * 1_000_003 + what) & 0x7FFFFFFF)


def _inputs(ws, seed, states=1):
    """States in reference order (a wet mid-event state, every storage x
    U(0.9, 1.1)), the forcing and the previous step's surface storage."""
    base = W.reference_state(ws, seed)
    ys = [W.jitter(base, 10 * seed + k) for k in range(states)]
    pcpdrp, edir, ett = W.random_forcing(ws, seed + 2)
    ws0 = ys[0][:ws.nelem] * _rng(seed, 1).uniform(0.5, 1.5, ws.nelem)
    return ys, pcpdrp, edir, ett, ws0


def _context(ws, inputs, stream=None):
    g = GpuRhs(ws, stream=stream)
    _, pcpdrp, edir, ett, ws0 = inputs
    g.set_forcing(pcpdrp, edir, ett)
    g.set_ws0_surf(ws0)
    return g


def _internal(g, y):
    """A reference-order host state on the device in the library's order."""
    a = torch.from_numpy(np.ascontiguousarray(y)).cuda()
    b = torch.empty_like(a)
    g.to_internal(a.data_ptr(), b.data_ptr())
    torch.cuda.synchronize()
    return b


def _vectors(n, seed):
    r = _rng(seed, 7)
    x = r.normal(0.0, 1e-3, n)                    # a correction
    y = r.uniform(0.0, 3.0, n)                    # storages (m)
    y[r.uniform(size=n) < 0.2] = 0.0              # dry surfaces
    v = r.normal(0.0, 1.0, n) / math.sqrt(n)      # a Krylov vector
    f = r.normal(0.0, 1e-6, n)                    # derivatives (m/s)
    return x, y, v, f


def _land_of(ws, case, seed):
    # January; every element with a leaf-area series and vegetation
    land = LAND.synthetic_land(ws, start=LAND_START, hours=LAND_HOURS, nstations=case["stations"], nlai=case["nlai"],
                               seed=seed)
    r = _rng(seed, 3)
    ne = ws.nelem
    land.params["lai_type"] = r.integers(1, case["nlai"] + 1, ne).astype(np.int32)
    cmc = r.uniform(0.0, 2e-4, ne)
    sneqv = np.where(r.uniform(size=ne) < 0.4, r.uniform(0.0, 0.03, ne), 0.0)
    return land, cmc, sneqv, LAND.epoch(LAND_START) + 3600 * (seed % 24) + 450


@functools.lru_cache(maxsize=2)
def _watersheds(systems, lo, hi):
    sizes = WL.log_uniform_sizes(systems, lo, hi, 0)
    return [W.generate(int(n), WL.river_count(int(n)), seed=k) for k, n in enumerate(sizes)]


def _solve_inputs(ws, steps, seed):
    y0 = W.jitter(W.relax_state(ws), seed, 0.98, 1.0)
    r = _rng(seed, 5)
    pcp = np.full(steps, r.uniform(0.5, 6.0) / 3.6e6)
    pet = r.uniform(0.05, 0.3) / 3.6e6
    return y0, pcp, np.full(steps, 0.3 * pet), np.full(steps, 0.7 * pet)


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "vec":
        lib = NV.load()
        n = case["n"]
        arrays = [torch.from_numpy(a).cuda() for a in _vectors(n, seed)] + [
            torch.empty(n, dtype=torch.float64, device="cuda") for _ in range(5)]
        first = lib.N_VNew_PihmGpu(n, None)  # the family: its stream and reduction workspace
        vs = []
        for a in arrays:
            v = lib.N_VCloneEmpty_PihmGpu(first)
            _set_array(lib, v, a.data_ptr())
            vs.append(v)
        lib.N_VDestroy_PihmGpu(first)
        return dict(kind=kind, lib=lib, n=n, arrays=arrays, vs=vs)
    if kind == "batch":
        wss = _watersheds(case["systems"], case["lo"], case["hi"])
        cases = []
        for k, ws in enumerate(wss):
            y0, pcp, edir, ett = _solve_inputs(ws, case["steps"], 1000 * seed + k)
            cases.append(dict(ws=ws, y0=y0, pcp=pcp, edir=edir, ett=ett, ctrl=StepControl(), outlet=-1))
        return dict(kind=kind, cases=cases, batch=Batch(limits_for(wss, case["steps"])))
    ws = _mesh(case["nelem"], case["mesh"], case.get("mode", 2))
    if kind == "solve":
        y0, pcp, edir, ett = _solve_inputs(ws, case["steps"], seed)
        m = GpuWatershed(ws, y0, pcp, edir, ett)
        m.g.set_diagnostics(False)
        return dict(kind=kind, m=m, y0=y0, steps=case["steps"], dry=np.zeros(3 * ws.nelem))
    inputs = _inputs(ws, seed, case.get("states", 1) if kind != "flux" else 3)
    ys = inputs[0]
    if kind == "host":
        return dict(kind=kind, g=_context(ws, inputs), y=ys[0], ydot=np.zeros(ws.neq))
    if kind == "ensemble":
        streams = [torch.cuda.Stream() for _ in range(case["contexts"])]
        ctx = [_context(ws, inputs, s.cuda_stream) for s in streams]
        yi = [_internal(_Ordered(ctx[0]), y) for y in ys]
        return dict(kind=kind, ctx=ctx, streams=streams, y=yi, ydot=[torch.empty_like(y) for y in yi],
                    out=[torch.empty_like(y) for y in yi])
    g = _context(ws, inputs)
    yi = [_internal(g, y) for y in ys]
    s = dict(kind=kind, g=g, y=yi, ydot=[torch.empty_like(yi[0]) for _ in range(case.get("steps", 1))],
             out=[torch.empty_like(yi[0]) for _ in range(case.get("steps", 1))])
    if kind == "land":
        land, cmc, sneqv, t = _land_of(ws, case, seed)
        g.land_init(land)
        g.land_set_state(cmc, sneqv)
        lo, hi = land.time_range()
        s.update(t=t, lo=lo, hi=hi - int(LSM_STEP))
    elif kind == "flux":
        params, state = NOAH.synthetic_noah(ws, seed=seed)
        g.noah_init(params, state)
        g.noah_set_forcing(NOAH.forcing(ws, 6 + seed % 12, seed=seed))
        g.noah_begin(yi[0].data_ptr())
    torch.cuda.synchronize()
    return s


class _Ordered:
    """to_internal of a context that has a stream of its own, done before it returns."""

    def __init__(self, g):
        self.g = g

    def to_internal(self, a, b):
        torch.cuda.synchronize()
        self.g.to_internal(a, b)


def _set_array(lib, v, ptr):
    f = lib.N_VSetArrayPointer_PihmGpu
    f.argtypes = [ctypes.c_void_p, ctypes.c_void_p]
    f.restype = None
    f(ptr, v)


def run(s):
    return _RUN[s["kind"]](s)


def _run_rhs(s):
    g = s["g"]
    g.rhs_device(s["y"][0].data_ptr(), s["ydot"][0].data_ptr())
    g.to_reference(s["ydot"][0].data_ptr(), s["out"][0].data_ptr())
    return s["out"][0]


def _run_host(s):
    rc = s["g"].rhs_host_ptr(s["y"].ctypes.data, s["ydot"].ctypes.data)
    if rc:
        raise RuntimeError(f"pihm_gpu_rhs_host returned {rc}")
    return s["ydot"]


def _run_ensemble(s):
    ctx, n = s["ctx"], len(s["ctx"])
    for k, (y, yd, o) in enumerate(zip(s["y"], s["ydot"], s["out"])):
        g = ctx[k % n]
        g.rhs_device(y.data_ptr(), yd.data_ptr())
        g.to_reference(yd.data_ptr(), o.data_ptr())
    return s["out"]


def _run_vec(s):
    """CVODE's error weights, a Newton correction's norm and update, and a
    modified Gram-Schmidt step, operation by operation."""
    lib = s["lib"]
    x, y, v, f, ewt, cor, res, w, z = s["vs"]
    lib.N_VAbs_PihmGpu(y, ewt)                      # CVEwtSetSS
    lib.N_VScale_PihmGpu(RELTOL, ewt, ewt)
    lib.N_VAddConst_PihmGpu(ewt, ABSTOL, ewt)
    lib.N_VInv_PihmGpu(ewt, ewt)
    lib.N_VLinearSum_PihmGpu(0.37, f, -1.25e-3, x, res)   # the Newton residual
    del_norm = lib.N_VWrmsNorm_PihmGpu(x, ewt)
    lib.N_VLinearSum_PihmGpu(1.0, y, 0.81, x, cor)        # the corrected state
    lib.N_VProd_PihmGpu(res, ewt, w)                # GMRES: scaled residual
    h = lib.N_VDotProd_PihmGpu(w, v)
    lib.N_VLinearSum_PihmGpu(1.0, w, -h, v, w)
    nrm = math.sqrt(lib.N_VDotProd_PihmGpu(w, w))
    lib.N_VScale_PihmGpu(1.0 / nrm, w, w)
    lib.N_VDiv_PihmGpu(w, ewt, z)
    top = lib.N_VMaxNorm_PihmGpu(z)
    return [a for a in s["arrays"][4:]] + [del_norm, h, nrm, top]


def _run_land(s):
    g, y = s["g"], s["y"][0].data_ptr()
    g.land_step(s["t"], LSM_STEP, y)
    s["t"] = s["t"] + int(LSM_STEP) if s["t"] + LSM_STEP <= s["hi"] else s["lo"]
    g.rhs_device(y, s["ydot"][0].data_ptr())
    g.to_reference(s["ydot"][0].data_ptr(), s["out"][0].data_ptr())
    return s["out"][0]


def _run_flux(s):
    g = s["g"]
    g.noah_step(3600.0)
    for k, (yd, o) in enumerate(zip(s["ydot"], s["out"])):
        y = s["y"][k % len(s["y"])].data_ptr()
        g.rhs_device(y, yd.data_ptr())
        g.noah_post_step(y, 60.0)
        g.to_reference(yd.data_ptr(), o.data_ptr())
    return s["out"]


def _run_solve(s):
    m = s["m"]
    lib, y0 = m.lib, s["y0"]
    if lib.N_VCopyFromHost_PihmGpu(m.scratch, y0.ctypes.data_as(ctypes.c_void_p)):
        raise RuntimeError("N_VCopyFromHost_PihmGpu failed")
    m.g.to_internal(lib.N_VGetDeviceArrayPointer_PihmGpu(m.scratch), m.device_state())
    m.g.set_ws0_surf(y0[:m.ws.nelem])
    m.g.set_river_edge_ovlflow(s["dry"])
    r = run_steps(m, StepControl(), s["steps"], m.set_forcing, record_every=s["steps"])
    return r["states"][-1], int(r["stats"].nst)


def _run_batch(s):
    b = s["batch"]
    ids = b.add_many(s["cases"])
    b.step()
    res = [b.result(i) for i in ids]
    for i in ids:
        b.release(i)
    return [np.concatenate([r["y"] for r in res]), np.array([r["stats"].nst for r in res])]


_RUN = dict(rhs=_run_rhs, host=_run_host, ensemble=_run_ensemble, vec=_run_vec, land=_run_land, flux=_run_flux,
            solve=_run_solve, batch=_run_batch)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
# Per element-evaluation: y, forcing and previous storage in, ydot out, the
# element's parameters and its share of the edges (332 B); per segment 184 B.
# The flops are the model's own double-precision operations, a power, a
# logarithm or a root counted as one.
def _rhs_work(nelem, times=1):
    nr = WL.river_count(nelem)
    return dict(bytes=times * (332.0 * nelem + 184.0 * nr), flops=times * (160.0 * nelem + 150.0 * nr))


def work(case):
    kind = case["kind"]
    if kind in ("rhs", "host"):
        return _rhs_work(case["nelem"])
    if kind == "ensemble":
        return _rhs_work(case["nelem"], case["states"])
    if kind == "vec":
        # inputs x, y, v, f and outputs ewt, corrected state, residual,
        # GMRES vector and scaled correction, once each
        n = float(case["n"])
        return dict(bytes=9 * 8 * n, flops=24 * n)
    if kind == "land":
        w = _rhs_work(case["nelem"])
        return dict(bytes=w["bytes"] + 260.0 * case["nelem"], flops=w["flops"] + 120.0 * case["nelem"])
    if kind == "flux":
        # Noah: 50 scalar planes and 9 of 4 layers in, about 30 scalars and 6 x 4
        # out; a post-step: 20 scalars and 7 of 4 layers in, 10 and 5 x 4 out
        w = _rhs_work(case["nelem"], case["steps"])
        ne = case["nelem"]
        return dict(bytes=w["bytes"] + 8.0 * ne * (140 + case["steps"] * 78),
                    flops=w["flops"] + ne * (2000.0 + case["steps"] * 300.0))
    if kind == "solve":
        # about 20 integrator steps of three evaluations and 80 vector operations
        ne, k = case["nelem"], case["steps"]
        w = _rhs_work(ne, 60 * k)
        return dict(bytes=w["bytes"] + k * 20 * 80 * 24.0 * 3 * ne, flops=w["flops"] + k * 20 * 80 * 2.0 * 3 * ne)
    sizes = WL.log_uniform_sizes(case["systems"], case["lo"], case["hi"], 0)
    ws = [work(dict(kind="solve", nelem=int(n), steps=case["steps"])) for n in sizes]
    return dict(bytes=sum(w["bytes"] for w in ws), flops=sum(w["flops"] for w in ws))


# ---------------------------------------------------------------------------
# the same results in plain numpy, 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind == "vec":
        return _exact_vec(case, seed)
    if kind not in ("rhs", "host", "ensemble", "land"):
        # the integrator's adaptive steps and Noah's column physics with its
        # inner iterations have no closed numpy form of this size
        return None
    ws = _mesh(case["nelem"], case["mesh"], case.get("mode", 2))
    ys, pcpdrp, edir, ett, ws0 = _inputs(ws, seed, case.get("states", 1))
    if kind == "land":
        pcpdrp, edir, ett = _np_land(ws, case, seed, ys[0])
    if kind != "ensemble":
        return _np_rhs(ws, ys[0], pcpdrp, edir, ett, ws0)[0]
    if case["nelem"] * case["states"] > 5_000_000:
        return None
    out, carry = [], [None] * case["contexts"]
    for k, y in enumerate(ys):  # a context keeps the river banks' overland flux from one evaluation to its next
        c = k % case["contexts"]
        d, carry[c] = _np_rhs(ws, y, pcpdrp, edir, ett, ws0, carry[c])
        out.append(d)
    return out


def _exact_vec(case, seed):
    x, y, v, f = _vectors(case["n"], seed)
    ewt = 1.0 / (RELTOL * np.abs(y) + ABSTOL)
    res = 0.37 * f - 1.25e-3 * x
    del_norm = math.sqrt(float(np.mean((x * ewt) ** 2)))
    cor = y + 0.81 * x
    w = res * ewt
    h = float(np.dot(w, v))
    w = w - h * v
    nrm = math.sqrt(float(np.dot(w, w)))
    w = w / nrm
    z = w / ewt
    return [ewt, cor, res, w, z, del_norm, h, nrm, float(np.max(np.abs(z)))]


DEPRSTG, GRADMIN, SATMIN, RIVGRADMIN, PSIMIN, GRAV = 1e-4, 5e-8, 0.1, 0.05, -70.0, 9.80665


def _avg_h(diff, here, there):
    return np.maximum(np.where(diff > 0.0, here, there), 0.0)


def _manning(h, grad, sf, crossa, rough):
    return crossa * np.power(h, 0.6666667) * grad / (np.sqrt(sf) * rough)


def _section(order, d, c):
    """Channel area and wetted perimeter at depth d."""
    area = np.select([order == 1, order == 2, order == 3],
                     [d * c, d * d / c, 4.0 * d * np.sqrt(d) / (3.0 * np.sqrt(c))],
                     3.0 * np.power(d, 4.0 / 3.0) / (2.0 * np.cbrt(c)))
    c13, c23 = np.cbrt(c), np.power(c, 2.0 / 3.0)
    perim = np.select(
        [order == 1, order == 2, order == 3],
        [2.0 * d + c, 2.0 * d * np.sqrt(1.0 + c * c) / c,
         np.sqrt(d * (1.0 + 4.0 * c * d) / c) + np.log(2.0 * np.sqrt(c * d) + np.sqrt(1.0 + 4.0 * c * d)) / (2.0 * c)],
        2.0 * (np.sqrt(d * (1.0 + 9.0 * c23 * d)) / 3.0
               + np.log(3.0 * c13 * np.sqrt(d) + np.sqrt(1.0 + 9.0 * c23 * d)) / (9.0 * c13)))
    return area, perim


def _np_rhs(ws, yv, pcpdrp, edir, ett, ws0, carry=None):
    """The PIHM right-hand side of one state, reference order; and the river
    banks' overland flux that the next evaluation's infiltration reads."""
    a = ws.arrays
    ne, nr = ws.nelem, ws.nriver
    pos = np.maximum(yv, 0.0)
    surf, unsat, gw = pos[:ne], pos[ne:2 * ne], pos[2 * ne:3 * ne]
    stage, rgw = pos[3 * ne:3 * ne + nr], pos[3 * ne + nr:]
    area, zmin, zmax, depth, dmac = a["area"], a["zmin"], a["zmax"], a["depth"], a["dmac"]
    with np.errstate(all="ignore"):
        surfh = np.where(surf <= 0.5 * DEPRSTG, np.sqrt(2.0 * DEPRSTG * surf), DEPRSTG + (surf - 0.5 * DEPRSTG))
        head = surfh + zmax
        k1 = a["kmach"] * a["areafv"] + a["ksath"] * (1.0 - a["areafv"])
        d2 = depth - dmac
        d1 = np.where(gw > depth, dmac, gw - d2)
        effk = np.where(gw > d2, (k1 * d1 + a["ksath"] * d2) / (d1 + d2), a["ksath"])
        nabr = a["nabr"]
        inner, bank = nabr > 0, nabr < 0
        kn = np.where(inner, nabr - 1, 0)
        sn = np.where(bank, -nabr - 1, 0)
        # water-surface gradient
        hj = np.where(inner, head[kn], np.where(
            bank, np.where(stage > a["riv_depth"], a["riv_zbed"] + stage, a["riv_zmax"])[sn], head[:, None]))

        def dh(l1, l2):
            return -(l1[:, 2] * (hj[:, 1] - hj[:, 0]) + l1[:, 1] * (hj[:, 0] - hj[:, 2]) + l1[:, 0] * (hj[:, 2] - hj[:, 1])) / (
                l2[:, 2] * (l1[:, 1] - l1[:, 0]) + l2[:, 1] * (l1[:, 0] - l1[:, 2]) + l2[:, 0] * (l1[:, 2] - l1[:, 1]))

        gx, gy = dh(a["nabr_y"], a["nabr_x"]), dh(a["nabr_x"], a["nabr_y"])
        gmag = np.sqrt(gx * gx + gy * gy)
        del gx, gy, hj
        # edge fluxes, each seen from its element
        ovl, sub = np.zeros((ne, 3)), np.zeros((ne, 3))
        for j in range(3):
            m = np.nonzero(inner[:, j])[0]
            k = kn[m, j]
            dist, edge = a["nabrdist"][m, j], a["edge"][m, j]
            diff = (gw[m] + zmin[m]) - (gw[k] + zmin[k])
            sub[m, j] = 0.5 * (effk[m] + effk[k]) * (diff / dist) * _avg_h(diff, gw[m], gw[k]) * edge
            diff = zmax[m] - zmax[k] if ws.surf_mode == 1 else head[m] - head[k]
            ah = _avg_h(diff, surfh[m] - DEPRSTG, surfh[k] - DEPRSTG)
            grad = diff / dist
            sf = np.where(grad > 0.0, grad, GRADMIN) if ws.surf_mode == 1 else np.maximum(0.5 * (gmag[m] + gmag[k]), GRADMIN)
            ovl[m, j] = _manning(ah, grad, sf, ah * edge, 0.5 * (a["rough"][m] + a["rough"][k]))
        # rivers
        down = a["down"]
        L, R = a["leftele"] - 1, a["rightele"] - 1
        go = down > 0
        dn = np.where(go, down - 1, 0)
        csa, per = _section(a["intrpl_ord"], stage, a["riv_coeff"])
        zbed, rzmin, rlen = a["riv_zbed"], a["riv_zmin"], a["riv_length"]
        dist = 0.5 * (rlen + rlen[dn])
        diff = zbed - zbed[dn] if ws.riv_mode == 1 else (stage + zbed) - (stage[dn] + zbed[dn])
        grad = diff / dist
        ap = 0.5 * (per + per[dn])
        ah = np.where(ap == 0.0, 0.0, 0.5 * (csa + csa[dn]) / ap)
        chan = _manning(ah, grad, np.where(grad > 0.0, grad, RIVGRADMIN), csa, 0.5 * (a["riv_rough"] + a["riv_rough"][dn]))
        grad = (zbed - (a["riv_node_zmax"] - a["riv_depth"])) / (0.5 * rlen)
        zero_grad = np.sqrt(grad) * csa * np.where(per > 0.0, np.power(csa / per, 2.0 / 3.0), 0.0) / a["riv_rough"]
        chan = np.where(go, chan, np.where(down == -3, zero_grad, csa * np.sqrt(GRAV * stage)))
        ke = 0.5 * (effk[L] + effk[R])
        diff = (rgw + rzmin) - (rgw[dn] + rzmin[dn])
        aquif = np.where(go, 0.5 * (ke + ke[dn]) * (diff / dist) * _avg_h(diff, rgw, rgw[dn])
                         * 0.5 * (a["riv_width"] + a["riv_width"][dn]), 0.0)
        f = {}
        for side, e, sd in (("l", L, a["riv_dist_left"]), ("r", R, a["riv_dist_right"])):
            bankz = np.maximum(a["riv_zmax"], zmax[e])
            eh, rh = zmax[e] + surfh[e], zbed + stage
            cw = a["riv_cwr"] * 2.0 * np.sqrt(2.0 * GRAV) * rlen / 3.0
            out = cw * np.where(eh > bankz, np.sqrt(rh - eh) * (rh - bankz), np.where(bankz < rh, np.sqrt(rh - bankz) * (rh - bankz), 0.0))
            into = -cw * np.where(rh > bankz, np.sqrt(eh - rh) * (eh - bankz), np.where(bankz < eh, np.sqrt(eh - bankz) * (eh - bankz), 0.0))
            f["ovl" + side] = np.where(rh > eh, out, np.where(surfh[e] > DEPRSTG, into, 0.0))
            above = zmin[e] > zbed
            partly = zmin[e] + gw[e] > zbed
            diff = rh - (gw[e] + zmin[e])
            h = _avg_h(diff, stage, np.where(above, gw[e], np.where(partly, zmin[e] + gw[e] - zbed, 0.0)))
            f["chan" + side] = rlen * 0.5 * (effk[e] + a["riv_ksath"]) * (diff / sd) * h
            diff = (rgw + rzmin) - (gw[e] + zmin[e])
            h = _avg_h(diff, rgw, np.where(above, 0.0, np.where(partly, zbed - zmin[e], gw[e])))
            f["sub" + side] = rlen * 0.5 * (effk[e] + ke) * (diff / sd) * h
        leak = a["riv_ksatv"] * a["riv_width"] * rlen * np.where(
            zbed - (rgw + rzmin) > 0.0, stage, stage + zbed - (rgw + rzmin)) / a["riv_bedthick"]
        up_c, up_a = np.zeros(nr), np.zeros(nr)
        np.subtract.at(up_c, dn[go], chan[go])
        np.subtract.at(up_a, dn[go], aquif[go])
        # vertical fluxes; infiltration sees the previous evaluation's flux on river edges
        old = np.zeros(2 * nr) if carry is None else carry
        left = L[sn] == np.arange(ne)[:, None]
        seen = np.where(bank, -np.where(left, old[:nr][sn], old[nr:][sn]), ovl)
        deficit = depth - gw
        shallow = gw > depth - a["dinf"]
        satn = np.clip(np.where(shallow, 1.0, unsat / np.where(shallow, 1.0, deficit)), SATMIN, 1.0)
        alpha, beta = a["alpha"], a["beta"]
        vm = beta / (beta - 1.0)
        t = 1.0 - np.power(1.0 - np.power(satn, vm), (beta - 1.0) / beta)
        kr = np.where(shallow, 1.0, np.sqrt(satn) * t * t)
        psi = -np.power(np.power(1.0 / satn, vm) - 1.0, 1.0 / beta) / alpha
        appl = np.maximum(-(seen / area[:, None]).sum(1), 0.0) + pcpdrp
        h_u = np.where(shallow, gw + zmin, np.maximum(psi, PSIMIN) + zmax - 0.5 * a["dinf"])
        dz = (surfh + zmax - h_u) / (0.5 * (surfh + a["dinf"]))
        dz = np.where((surfh <= 0.0) & (dz > 0.0), 0.0, dz)
        kinfv, kmacv, fh = a["kinfv"], a["kmacv"], a["areafh"]
        mat, mac = kinfv * (1.0 - fh) * kr, kmacv * fh
        t2 = 1.0 - np.sqrt(1.0 - satn * satn)
        kinf = np.select([fh == 0.0, surfh > DEPRSTG, appl <= dz * kinfv * kr, appl < dz * (mac + mat)],
                         [kinfv * kr, mat + mac, kinfv * kr, mat + mac * np.sqrt(satn) * t2 * t2], mat + mac)
        infil = kinf * dz
        infil = np.where(shallow, infil, np.maximum(infil, 0.0))
        infil = np.minimum(infil, appl + np.maximum(ws0, 0.0) / ws.stepsize) * np.clip(surfh / DEPRSTG, 0.0, 1.0)
        infil = np.where(unsat + gw > depth, 0.0, infil)
        ksv = a["ksatv"]
        deep = deficit > dmac
        k2 = np.where(deep, kr * ksv, np.where(fh > 0.0, kmacv * fh + ksv * (1.0 - fh), ksv))
        d1 = np.where(deep, dmac, deficit)
        d2 = np.where(deep, deficit - dmac, dmac - deficit)
        d3 = np.where(deep, gw, gw - (dmac - deficit))
        rechg = (kr * ksv * d1 + k2 * d2 + ksv * d3) / (d1 + d2 + d3) * (0.5 * deficit + psi) / (0.5 * (deficit + gw))
        rechg = np.where((rechg > 0.0) & (unsat <= 0.0), 0.0, rechg)
        rechg = np.where((rechg < 0.0) & (gw <= 0.0), 0.0, rechg)
        rechg = np.where(shallow, infil, rechg)
        # evapotranspiration's store, then the rows
        ponded = surfh >= DEPRSTG
        e_s, e_g = np.where(ponded, edir, 0.0), np.where(~ponded & shallow, edir, 0.0)
        e_u = edir - e_s - e_g
        t_g = np.where(gw > depth - a["rzd"], ett, 0.0)
        t_u = ett - t_g
        now = np.where(left, f["ovll"][sn], f["ovlr"][sn])
        seep = np.where(left, (f["chanl"] + f["subl"])[sn], (f["chanr"] + f["subr"])[sn])
        ovl, sub = np.where(bank, -now, ovl), np.where(bank, -seep, sub)
        ds = pcpdrp - infil - e_s - (ovl / area[:, None]).sum(1)
        du = (infil - rechg - e_u - t_u) / a["porosity"]
        dg = (rechg - e_g - t_g - (sub / area[:, None]).sum(1)) / a["porosity"]
        ra = a["riv_area"]
        dst = -(up_c + chan + f["ovll"] + f["ovlr"] + f["chanl"] + f["chanr"] + leak) / ra
        drg = (-f["subl"] - f["subr"] - aquif - up_a + leak) / (a["riv_porosity"] * ra)
    return np.concatenate([ds, du, dg, dst, drg]), np.concatenate([f["ovll"], f["ovlr"]])


# monthly roughness length (January) of the land types the generator draws,
# and January's degree-day melt factor: the model's climatology
_Z0_JAN = {1: 0.5, 2: 0.5, 3: 0.5, 4: 0.5, 5: 0.2, 6: 0.01, 7: 0.01, 8: 0.01, 9: 0.15, 10: 0.1, 12: 0.05, 13: 0.5,
           14: 0.05, 16: 0.01}
_MELT_JAN = 0.001308019


def _np_land(ws, case, seed, yv):
    """pcpdrp, edir and ett after one land-surface step: the forcing series
    interpolated, snow, interception, Penman-Monteith evapotranspiration."""
    land, cmc, sneqv, t = _land_of(ws, case, seed)
    p, a = land.params, ws.arrays
    ne, dt = ws.nelem, LSM_STEP

    def series(lens, times, data):
        out, o = [], 0
        for n in lens:
            tt, d = times[o:o + n], data[o:o + n]
            k = int(np.searchsorted(tt, t))
            out.append(((tt[k] - t) * d[k - 1] + (t - tt[k - 1]) * d[k]) / float(tt[k] - tt[k - 1]))
            o += n
        return np.array(out)

    met = series(land.meteo_len, land.meteo_time, land.meteo_data)[p["meteo_type"] - 1]
    lai = series(land.lai_len, land.lai_time, land.lai_data)[p["lai_type"] - 1]
    z0 = np.zeros(41)
    for k, v in _Z0_JAN.items():
        z0[k] = v
    z0 = z0[p["lc_type"]]
    prcp, tc, rh, wind, sol = met[:, 0] / 1000.0, met[:, 1] - 273.15, met[:, 2] / 100.0, met[:, 3], np.maximum(met[:, 4], 0.0)
    with np.errstate(all="ignore"):
        radnet = sol * (1.0 - 0.5 * (p["albedomin"] + p["albedomax"]))
        vp = 611.2 * np.exp(17.67 * tc / (tc + 243.5)) * rh
        pres = 101.325e3 * np.power((293.0 - 0.0065 * a["zmax"]) / 293.0, 5.26)
        qv, qs = 0.622 * vp / pres, 0.622 * (vp / rh) / pres
        frac = np.where(tc < -3.0, 1.0, np.where(tc > 1.0, 0.0, (1.0 - tc) / 4.0))
        sneqv = sneqv + frac * prcp * dt
        melt = np.where(tc > 0.0, tc * _MELT_JAN, 0.0)
        melt = np.where(sneqv > melt * dt, melt, sneqv / dt)
        shd = p["shdfac"]
        cap = p["cmcfactr"] * lai * shd
        ra = np.log(p["zlvl_wind"] / z0) * np.log(10.0 * p["zlvl_wind"] / z0) / (wind * 0.16)
        tk = tc + 273.15
        gamma = 4.0 * 0.7 * 5.67e-8 * 287.04 / 1004.0 * tk ** 4 / (pres / ra) + 1.0
        delta = 2.501e6 * 2.501e6 * 0.622 / 461.5 / 1004.0 / (tk * tk) * qs
        etp = (radnet * delta + gamma * (1.2 * 2.501e6 * (qs - qv) / ra)) / (1000.0 * 2.501e6 * (delta + gamma))
        unsat, gw = yv[ne:2 * ne], yv[2 * ne:3 * ne]
        r = unsat / (a["depth"] - gw)
        satn = np.where(r > 1.0, 1.0, np.where(r < 0.0, 0.0, 0.5 * (1.0 - np.cos(3.14 * r))))
        satn = np.where(a["depth"] - gw < a["rzd"], 1.0, satn)
        betas = np.clip((satn * a["porosity"] + p["smcmin"] - p["smcwlt"]) / (p["smcref"] - p["smcwlt"]), 1e-4, 1.0)
        edir = np.maximum((1.0 - shd) * betas * betas * etp, 0.0)
        wet = np.clip(cmc, 0.0, cap) / cap
        pw = np.power(wet, p["cfactr"])
        ec = np.maximum(shd * pw * etp, 0.0)
        fr = np.maximum(1.1 * radnet / (p["rgl"] * lai), 0.0)
        al = np.minimum((1.0 + fr) / (fr + p["rsmin"] / p["rsmax"]), 1e4)
        et = np.maximum(1.0 - 0.0016 * (p["topt"] - 273.15 - tc) ** 2, 1e-4)
        gs = np.maximum(1.0 / (1.0 + 0.00025 * (vp / rh - vp)), 0.01)
        rs = np.minimum(p["rsmin"] * al / (betas * lai * et * gs), p["rsmax"])
        pc = (1.0 + delta / gamma) / (1.0 + rs / ra + delta / gamma)
        ett = np.maximum(shd * pc * (1.0 - pw) * etp, 0.0)
        ett = np.where((gw < a["depth"] - a["rzd"]) & (unsat <= 0.0), 0.0, ett)
        drip = np.where(cmc <= 0.0, 0.0, 6.52e-7 * cap * np.exp(3.89 * cmc / cap))
        drip = np.where(drip * dt > cmc, cmc / dt, drip)
        fall = (1.0 - frac) * prcp * shd * dt
        left = cmc + fall - ec * dt - drip * dt
        # an empty canopy shares what it had between evaporation and drip
        ec2 = ec / (ec + drip) * fall
        drip = np.where(left > cap, drip + (left - cap) / dt,
                        np.where((left < 0.0) & (ec + drip > 0.0), drip / (ec2 + drip) * fall, drip))
        pcpdrp = (1.0 - shd) * (1.0 - frac) * prcp + drip + melt
    return pcpdrp, edir, ett
