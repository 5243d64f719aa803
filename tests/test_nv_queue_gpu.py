"""The integrator's queued element-wise operations and the reductions that end
them (one kernel) against the same integration with every operation issued
through the vectors' own table: the same bits and the same counters, around
the lengths where the kernel's layout changes (a warp, a block of the
reduction order, its spread form's last length, one pass over the vector)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

VP, D = ctypes.c_void_p, ctypes.c_double
OPS = ["nvgetvectorid", "nvclone", "nvcloneempty", "nvdestroy", "nvspace", "nvgetarraypointer", "nvsetarraypointer",
       "nvlinearsum", "nvconst", "nvprod", "nvdiv", "nvscale", "nvabs", "nvinv", "nvaddconst", "nvdotprod", "nvmaxnorm",
       "nvwrmsnorm", "nvwrmsnormmask", "nvmin"]
RHS = ctypes.CFUNCTYPE(ctypes.c_int, D, VP, VP, VP)


class Ops(ctypes.Structure):
    _fields_ = [(n, VP) for n in OPS]


class Vec(ctypes.Structure):
    _fields_ = [("content", VP), ("ops", ctypes.POINTER(Ops))]


def _table(lib):
    """Pass-through replacements of the table's operations, as a caller that
    counts or traces them installs; clones get them too."""
    keep = {}

    def install(v):
        ops = ctypes.cast(v, ctypes.POINTER(Vec)).contents.ops.contents
        for name, f in keep.items():
            setattr(ops, name, ctypes.cast(f, VP))
        return v

    vec = dict(nvlinearsum=("N_VLinearSum_PihmGpu", None, [D, VP, D, VP, VP]),
               nvconst=("N_VConst_PihmGpu", None, [D, VP]), nvprod=("N_VProd_PihmGpu", None, [VP] * 3),
               nvdiv=("N_VDiv_PihmGpu", None, [VP] * 3), nvscale=("N_VScale_PihmGpu", None, [D, VP, VP]),
               nvabs=("N_VAbs_PihmGpu", None, [VP] * 2), nvinv=("N_VInv_PihmGpu", None, [VP] * 2),
               nvaddconst=("N_VAddConst_PihmGpu", None, [VP, D, VP]), nvdotprod=("N_VDotProd_PihmGpu", D, [VP] * 2),
               nvmaxnorm=("N_VMaxNorm_PihmGpu", D, [VP]), nvwrmsnorm=("N_VWrmsNorm_PihmGpu", D, [VP] * 2),
               nvmin=("N_VMin_PihmGpu", D, [VP]))
    for name, (sym, res, args) in vec.items():
        inner = ctypes.CFUNCTYPE(res, *args)((sym, lib))
        keep[name] = ctypes.CFUNCTYPE(res, *args)(lambda *a, inner=inner: inner(*a))
    clone = ctypes.CFUNCTYPE(VP, VP)(("N_VClone_PihmGpu", lib))
    keep["nvclone"] = ctypes.CFUNCTYPE(VP, VP)(lambda w: install(clone(w)))
    return install, keep


def _solve(lib, n, wrapped, deferred, two_families):
    from pihm_gpu.solver import BdfStats
    rng = np.random.default_rng(n)
    put = lambda v, a: lib.N_VCopyFromHost_PihmGpu(v, a.ctypes.data_as(ctypes.POINTER(D)))  # noqa: E731
    y = lib.N_VNew_PihmGpu(n, None)
    yout = lib.N_VNew_PihmGpu(n, None) if two_families else lib.N_VClone_PihmGpu(y)
    k = lib.N_VClone_PihmGpu(y)
    if wrapped:
        install, keep = _table(lib)
        for v in (y, yout):
            install(v)
    assert put(y, rng.uniform(0.5, 2.0, n)) == 0 and put(k, -np.exp(rng.uniform(-3.0, 3.0, n))) == 0

    # y' = -k y^2, entry by entry, through the library's own operations
    def f(t, yy, ydot, ud):
        lib.N_VProd_PihmGpu(yy, yy, ydot)
        lib.N_VProd_PihmGpu(ydot, k, ydot)
        return 0

    cb = RHS(f)
    m = lib.pihm_bdf_create()
    try:
        assert lib.pihm_bdf_init(m, ctypes.cast(cb, VP), 0.0, y) == 0
        assert lib.pihm_bdf_ss_tolerances(m, 1e-5, 1e-7) == 0
        assert lib.pihm_bdf_set_stab_lim_det(m, 1) == 0
        assert lib.pihm_bdf_set_deferred_scalars(m, deferred) == 0
        t, states = D(0.0), []
        for tout in (0.5, 2.0):
            assert lib.pihm_bdf_solve(m, tout, yout, ctypes.byref(t)) == 0
            out = np.empty(n)
            assert lib.N_VCopyToHost_PihmGpu(yout, out.ctypes.data_as(ctypes.POINTER(D))) == 0
            states.append(out)
        s = BdfStats()
        assert lib.pihm_bdf_get_stats(m, ctypes.byref(s)) == 0
        return states, [getattr(s, name) for name, _ in s._fields_]
    finally:
        lib.pihm_bdf_free(m)
        for v in (k, yout, y):
            lib.N_VDestroy_PihmGpu(v)


@pytest.mark.parametrize("n", [1, 31, 33, 1023, 1025, 4097, 131_072, 131_073, 622_592, 622_593])
def test_queued_operations_same_solve(n):
    from pihm_gpu import nvector, solver
    lib = solver._bind(nvector.load())
    ref = _solve(lib, n, True, 0, False)
    assert ref[1][0] > 10 and ref[1][5] > 0  # steps, GMRES iterations
    for deferred, two in ((0, False), (1, True)):
        got = _solve(lib, n, False, deferred, two)
        assert got[1] == ref[1]
        for a, b in zip(got[0], ref[0]):
            assert np.array_equal(a, b)
