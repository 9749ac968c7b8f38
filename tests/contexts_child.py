"""Child process of tests/test_gpu_contexts.py: library calls from the device's primary context and from a
context of the application's own, in turn, as a program does that embeds the library beside its own driver
API code.  No torch is loaded.

    python contexts_child.py alternate | trim | destroy     -> one JSON line on stdout
"""
import ctypes as C
import json
import sys
from pathlib import Path

import numpy as np

sys.path.insert(0, str(Path(__file__).resolve().parent.parent))

from dogpup_b200 import _lib  # noqa: E402
from dogpup_b200._lib import lib  # noqa: E402  (loads libdogpup_b200.so)

U64, VP, SZ = C.c_uint64, C.c_void_p, C.c_size_t
cu = C.CDLL("libcuda.so.1")
cu.cuInit.argtypes = [C.c_uint]
cu.cuDeviceGet.argtypes = [C.POINTER(C.c_int), C.c_int]
cu.cuCtxCreate_v2.argtypes = [C.POINTER(VP), C.c_uint, C.c_int]
cu.cuCtxDestroy_v2.argtypes = [VP]
cu.cuCtxSetCurrent.argtypes = [VP]
cu.cuCtxGetCurrent.argtypes = [C.POINTER(VP)]
cu.cuDevicePrimaryCtxRetain.argtypes = [C.POINTER(VP), C.c_int]
cu.cuMemAlloc_v2.argtypes = [C.POINTER(U64), SZ]
cu.cuMemFree_v2.argtypes = [U64]
cu.cuMemcpyHtoD_v2.argtypes = [U64, VP, SZ]
cu.cuMemcpyDtoH_v2.argtypes = [VP, U64, SZ]
cu.cuMemGetInfo_v2.argtypes = [C.POINTER(SZ), C.POINTER(SZ)]


def ck(rc, what):
    if rc != 0:
        raise RuntimeError(f"{what}: {rc}")


def up(a):
    a = np.ascontiguousarray(a)
    p = U64()
    ck(cu.cuMemAlloc_v2(C.byref(p), a.nbytes), "cuMemAlloc")
    ck(cu.cuMemcpyHtoD_v2(p, a.ctypes.data_as(VP), a.nbytes), "cuMemcpyHtoD")
    return p


def down(p, like):
    ck(cu.cuMemcpyDtoH_v2(like.ctypes.data_as(VP), p, like.nbytes), "cuMemcpyDtoH")
    return like


def free_bytes():
    f, t = SZ(), SZ()
    ck(cu.cuMemGetInfo_v2(C.byref(f), C.byref(t)), "cuMemGetInfo")
    return f.value


def lm_update(jt, y):
    """One LM update in the current context; its buffers live only here."""
    nv, nm = jt.shape
    bufs = [up(jt), up(y), up(np.zeros(nv))]
    form = C.c_int32()
    ck(lib.dgp_lm_update(VP(bufs[0].value), nv, nm, None, VP(bufs[1].value), 0.1, VP(bufs[2].value), 0, C.byref(form),
                         None), "dgp_lm_update")
    x = down(bufs[2], np.empty(nv))
    for b in bufs:
        ck(cu.cuMemFree_v2(b), "cuMemFree")
    return x


def matrix(n=20000, band=12):
    """A diagonally dominant banded K and M in CSR form."""
    cols = np.arange(n)[:, None] + np.arange(-band, band + 1)
    keep = (cols >= 0) & (cols < n)
    rp = np.concatenate([[0], np.cumsum(keep.sum(1))]).astype(np.int32)
    off = np.broadcast_to(np.abs(np.arange(-band, band + 1)), cols.shape)
    k = np.where(off == 0, 2.0 * band + 1.0, -1.0 / np.maximum(off, 1))
    return rp, cols[keep].astype(np.int32), k[keep], np.where(off == 0, 1.0, 0.0)[keep]


def plan_and_solve(nf=16, ns=16):
    """A solver plan in the current context and its first solve; (handle, buffers)."""
    rp, col, K, M = matrix()
    n = len(rp) - 1
    bufs = [up(rp), up(col), up(K), up(M)]
    h = VP()
    ck(lib.dgp_solver_create(C.byref(h), *[VP(b.value) for b in bufs[:2]], n, len(col), *[VP(b.value) for b in bufs[2:]],
                             0.1, nf, ns, None, None), "dgp_solver_create")
    nodes, w = np.arange(4 * ns, dtype=np.int32) * 300, np.full(4 * ns, 0.25)
    fpsf = np.tile([1.0, 0.0], nf)
    bufs += [up(nodes), up(w), up(fpsf), up(np.zeros(2 * nf * n * ns))]
    opts, rep = _lib.default_opts(), _lib.SolveReport()
    opts.precision, opts.tol = _lib.PREC_MIXED, 1e-8
    ck(lib.dgp_solve_sources(h, *[VP(b.value) for b in bufs[4:7]], ns, VP(bufs[7].value), C.byref(opts), C.byref(rep),
                             None), "dgp_solve_sources")
    for b in bufs:
        ck(cu.cuMemFree_v2(b), "cuMemFree")
    return h


def trim(prim, destroy_in):
    """Free memory before a plan, with it, after it is destroyed (in the given context), and after the trim."""
    ck(cu.cuCtxSetCurrent(prim), "cuCtxSetCurrent")
    ck(lib.dgp_solver_destroy(plan_and_solve()), "dgp_solver_destroy")   # modules loaded, pools made
    ck(lib.dgp_trim_memory(), "dgp_trim_memory")
    free = [free_bytes()]
    h = plan_and_solve()
    free.append(free_bytes())
    ck(cu.cuCtxSetCurrent(destroy_in), "cuCtxSetCurrent")
    ck(lib.dgp_solver_destroy(h), "dgp_solver_destroy")
    cur = VP()
    ck(cu.cuCtxGetCurrent(C.byref(cur)), "cuCtxGetCurrent")
    assert cur.value == destroy_in.value
    ck(cu.cuCtxSetCurrent(prim), "cuCtxSetCurrent")
    free.append(free_bytes())
    ck(lib.dgp_trim_memory(), "dgp_trim_memory")
    return free + [free_bytes()]


def main():
    ck(cu.cuInit(0), "cuInit")
    dev, prim, own = C.c_int(), VP(), VP()
    ck(cu.cuDeviceGet(C.byref(dev), 0), "cuDeviceGet")
    ck(cu.cuDevicePrimaryCtxRetain(C.byref(prim), dev), "cuDevicePrimaryCtxRetain")
    ck(cu.cuCtxCreate_v2(C.byref(own), 0, dev), "cuCtxCreate")
    if sys.argv[1] != "alternate":
        print(json.dumps({"free": trim(prim, own if sys.argv[1] == "destroy" else prim)}))
        return
    rng = np.random.default_rng(1)
    jt, y = rng.standard_normal((2500, 1500)).astype(np.float32), rng.standard_normal(1500)
    xs, free = [], []
    for _ in range(10):
        for ctx in (prim, own):
            ck(cu.cuCtxSetCurrent(ctx), "cuCtxSetCurrent")
            xs.append(lm_update(jt, y))
        free.append(free_bytes())
    J = jt.T.astype(float)
    H = J.T @ J
    ref = np.linalg.solve(H + 0.1 * H.diagonal().max() * np.eye(H.shape[0]), J.T @ y)
    print(json.dumps({"free": free, "err": [float(np.linalg.norm(x - ref) / np.linalg.norm(ref)) for x in xs]}))
    ck(cu.cuCtxDestroy_v2(own), "cuCtxDestroy")


if __name__ == "__main__":
    main()
