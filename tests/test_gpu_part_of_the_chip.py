"""Solves on a stream whose context has a part of the SMs (a green context): a launch of one block for
every SM of the device does not fit there, and a kernel for each phase takes its place."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

RESOURCE = 144                   # bytes of a CUdevResource, whose SM count is at offset 96


@pytest.fixture
def half_stream():
    """A stream of a context with 64 SMs."""
    import torch
    torch.zeros(1, device="cuda")
    cu = ctypes.CDLL("libcuda.so.1")
    if not all(hasattr(cu, f) for f in ("cuDeviceGetDevResource", "cuGreenCtxCreate", "cuGreenCtxStreamCreate")):
        pytest.skip("the driver has no green contexts")

    def call(fn, *args):
        rc = getattr(cu, fn)(*args)
        if rc:
            pytest.skip("%s: driver error %d" % (fn, rc))

    every, some, rest = ((ctypes.c_ubyte * RESOURCE)() for _ in range(3))
    groups, desc, ctx, stream = ctypes.c_uint(1), ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()
    call("cuDeviceGetDevResource", 0, ctypes.byref(every), 1)                      # SMs
    call("cuDevSmResourceSplitByCount", ctypes.byref(some), ctypes.byref(groups), ctypes.byref(every),
         ctypes.byref(rest), 0, 64)
    call("cuDevResourceGenerateDesc", ctypes.byref(desc), ctypes.byref(some), 1)
    call("cuGreenCtxCreate", ctypes.byref(ctx), desc, 0, 1)
    call("cuGreenCtxStreamCreate", ctypes.byref(stream), ctx, 1, 0)                # non-blocking
    yield stream
    cu.cuStreamSynchronize(stream)
    cu.cuStreamDestroy_v2(stream)
    cu.cuGreenCtxDestroy(ctx)


def test_plain_solves(half_stream):
    import torch
    from pybella_gb300 import _lib, workloads
    w = workloads.rising_bubble_member((160, 80), 2.0, 0.0)
    A = workloads.operator_2d(w)
    x = torch.zeros(A.n, dtype=torch.float64, device="cuda")
    lib = A.ws._lib
    for entry, precision in (("bella_bicgstab", 0), ("bella_bicgstab", 1), ("bella_bicgstab", 2),
                             ("bella_bicgstab2d_noalloc", 0)):
        x.zero_()
        torch.cuda.synchronize()
        o, st = _lib.SolveOpts(), _lib.SolveStats()
        lib.bella_solve_opts_default(ctypes.byref(o))
        o.precision, o.tol, o.maxiter = precision, 1e-8, 6000
        first = ctypes.byref(A._op) if entry.endswith("noalloc") else A.ws.handle
        rc = getattr(lib, entry)(first, w["b"].data_ptr(), x.data_ptr(), ctypes.byref(o), ctypes.byref(st), half_stream)
        assert rc == 0 and st.status == 0 and st.iterations > 64, (entry, precision, rc)
        torch.cuda.synchronize()
        r = w["b"] - A.matvec(x)
        assert float(torch.linalg.norm(r)) <= 1.01e-8 * float(torch.linalg.norm(w["b"]))
