"""Performance cases: the work a diffuse-optics program has this framework do.

Each case is one call (or one short chain of calls) a program repeats: a forward
model after a property update, a loss gradient, a sensitivity, an LM update, a
batch of meshes.  The mesh, its optodes and the voxel basis are set up once per
geometry and kept, as such a program keeps them; the seed gives the optical
properties, fields, data and weights.  `exact` restates each result in 64-bit
torch: P1 assembly, a Jacobi-preconditioned Krylov solve, dense contractions.
"""
import ctypes
import functools
import math

import numpy as np
import scipy.sparse as sp
import torch

from dogpup_b200 import api, meshgen, workloads
from dogpup_b200._lib import check, lib
from dogpup_b200.autograd import TimeGatedForward
from dogpup_b200.batch import UnevenBatch

C_MEDIUM = 2.99792458e11 / 1.4  # mm/s
T_AXIS = workloads.time_axis(10e-9)
NT = len(T_AXIS)


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a first look at one small phantom: default precision and tolerance, every launch counts
        dict(name="forward small fp64", kind="forward", shape="cylinder", size=16.0, h=1.5, ns=8, nd=8, nf=8,
             precision="fp64", tol=1e-12),
        # the plain FP64 forward model of a 55k-node cylinder, 16 + 16 optodes, 32 harmonics
        dict(name="forward cylinder fp64", kind="forward", shape="cylinder", size=60.0, h=1.5, ns=16, nd=16, nf=32,
             precision="fp64", tol=1e-12),
        # a few sources on a mid-size head: ragged source and harmonic counts, mixed precision
        dict(name="forward ragged mixed", kind="forward", shape="ellipsoid", size=60.0, h=1.4, ns=11, nd=7, nf=21,
             precision="mixed", tol=1e-12),
        # the production forward model: 101,880-node head, 32 sources x 64 harmonics, mixed precision
        dict(name="forward head mixed", kind="forward", shape="ellipsoid", size=90.0, h=1.38, ns=32, nd=32, nf=64,
             precision="mixed", tol=1e-12),
        # one step of a gradient-based fit: time-gated data and dL/dmua, dL/dmusp through the autograd function
        dict(name="gradient cylinder mixed", kind="gradient", shape="cylinder", size=40.0, h=1.6, ns=16, nd=16,
             nf=32, ng=10, precision="mixed", tol=1e-12),
        # the explicit time-gated Jacobian on the nodes of the head, 1,024 links x 20 gates
        dict(name="tg jacobian nodes", kind="jac_tg", shape="ellipsoid", size=90.0, h=1.38, ns=32, nd=32, nf=64,
             ng=20, pitch=0.0, rytov=False),
        # the Jacobian of an LM iteration: voxel basis, Rytov-normalised, 10 gates
        dict(name="tg jacobian voxels", kind="jac_tg", shape="cylinder", size=60.0, h=1.5, ns=32, nd=32, nf=32,
             ng=10, pitch=2.0, rytov=True),
        # the reverse mode of the same map: J^T g on the nodes without forming J
        dict(name="tg vjp nodes", kind="jac_vjp", shape="ellipsoid", size=90.0, h=1.38, ns=32, nd=32, nf=64, ng=20,
             pitch=0.0, rytov=False),
        # the frequency-domain Jacobian on a coarse voxel grid
        dict(name="complex jacobian voxels", kind="jac_fd", shape="cylinder", size=60.0, h=1.5, ns=16, nd=15, nf=32,
             pitch=3.5),
        # the LM update with fewer measurements than voxels (2 mm voxels) ...
        dict(name="lm update fine voxels", kind="lm", nv=22971, nm=10240, lam=0.01, weighted=True),
        # ... and with more measurements than voxels (odd sizes, unweighted)
        dict(name="lm update coarse voxels", kind="lm", nv=3333, nm=7001, lam=0.01, weighted=False),
        # meshes of different sizes, source and harmonic counts in one batch: forward, adjoint and vjp of each
        dict(name="uneven batch", kind="batch", count=4, size=24.0, growth=1.3, h=1.5, ns=8, nf=16, ng=10,
             tol=1e-12),
    ]


def _spread(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _draw_mesh(rng, most):
    """A shape whose node count stays near or below `most`."""
    shape = rng.choice(("cylinder", "ellipsoid"))
    h = round(rng.uniform(1.35, 2.1), 3)
    nodes = _spread(rng, 2000, most)
    volume = nodes * h ** 3 * 0.93
    # cylinder: radius size/2, height size; ellipsoid: axes size x (1, 5/6, 7/9)
    fill = math.pi / 4 if shape == "cylinder" else math.pi / 6 * 5 / 6 * 7 / 9
    return dict(shape=shape, size=round((volume / fill) ** (1 / 3), 2), h=h)


def draw(rng):
    kind = rng.choice(("forward", "forward", "forward", "gradient", "jac_tg", "jac_tg", "jac_vjp", "jac_fd", "lm",
                       "lm", "batch"))
    if kind == "lm":
        nv, nm = int(_spread(rng, 300, 22000)), int(_spread(rng, 300, 10000))
        return dict(kind=kind, nv=nv, nm=nm if min(nv, nm) <= 10000 else 10000, lam=round(_spread(rng, 3e-3, 0.1), 4),
                    weighted=rng.random() < 0.5)
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(2, 4), size=round(rng.uniform(16, 24), 2),
                    growth=round(rng.uniform(1.1, 1.3), 2), h=round(rng.uniform(1.5, 2.0), 3), ns=rng.randint(3, 8),
                    nf=rng.randint(6, 16), ng=rng.randint(4, 12), tol=1e-12)
    ns, nd = int(_spread(rng, 3, 49)), int(_spread(rng, 3, 49))
    if kind in ("forward", "gradient"):
        precision = rng.choice(("fp64", "mixed", "mixed"))
        nf = int(_spread(rng, 4, 65))
        most = (2.5e7 if precision == "fp64" else 1.2e8) / (ns * nf) / (2 if kind == "gradient" else 1)
        c = dict(kind=kind, **_draw_mesh(rng, max(2500, min(90000, most))), ns=ns, nd=nd, nf=nf)
        if kind == "gradient":
            c["ng"] = rng.randint(4, 20)
        return dict(c, precision=precision, tol=1e-12)
    nf, ng = int(_spread(rng, 8, 97)), rng.randint(4, 24)
    if kind == "jac_fd":
        return dict(kind=kind, **_draw_mesh(rng, min(50000, 2.5e9 / (nf * ns * nd))), ns=ns, nd=nd, nf=nf,
                    pitch=round(rng.uniform(3.5, 5.0), 2))
    c = dict(kind=kind, **_draw_mesh(rng, min(50000, 1e11 / (ns * nd * nf * ng))), ns=ns, nd=nd, nf=nf, ng=ng)
    voxels = rng.random() < 0.5
    return dict(c, pitch=round(rng.uniform(2.0, 4.0), 2) if voxels else 0.0, rytov=rng.random() < 0.5)


# ------------------------------------------------------- geometry, kept per mesh
def _ring(n, shape, size, phase):
    """n optodes on the surface: one ring up to 16 of them, else rings of about 16."""
    rings = max(1, -(-n // 16))
    out = []
    for q in range(rings):
        m = n // rings + (q < n % rings)
        z = size / 2 + size * 0.12 * (q - (rings - 1) / 2) if shape == "cylinder" else \
            size * 7 / 18 * 0.3 * (q - (rings - 1) / 2)
        if shape == "cylinder":
            a, b = size / 2, size / 2
        else:
            s = math.sqrt(1 - (z / (size * 7 / 18)) ** 2)
            a, b = size / 2 * s, size * 5 / 12 * s
        out.append(workloads.ring(m, np.zeros(3), (a, b), z, phase=phase + 0.4 * q))
    return np.concatenate(out)


@functools.lru_cache(maxsize=6)
def _tetmesh(shape, size, h):
    if shape == "cylinder":
        return meshgen.cylinder_mesh(size / 2, size, h, jitter=0.13 * h, seed=1)
    return meshgen.ellipsoid_mesh((size, size * 5 / 6, size * 7 / 9), h, jitter=0.13 * h, seed=1)


@functools.lru_cache(maxsize=5)
def _dmesh(shape, size, h, ns, nd, nf):
    """The program's mesh: topology, optodes and, after its first solve, the solver plan."""
    m = _tetmesh(shape, size, h)
    return workloads.build_dmesh(dict(
        mesh=m, mua=np.full(m.nn, 0.01), musp=np.full(m.nn, 1.0), nr=1.4, src=_ring(ns, shape, size, 0.0),
        det=_ring(nd, shape, size, math.pi / max(ns, nd)), link=workloads.all_pairs(ns, nd), t=T_AXIS, nf=nf))


@functools.lru_cache(maxsize=4)
def _voxels(shape, size, h, pitch):
    """Mesh-to-voxel interpolation of a cubic voxel grid: barycentric weights in the mesh's lattice."""
    m = _tetmesh(shape, size, h)
    lo, hi = m.node.min(0), m.node.max(0)
    ax = [np.arange(lo[d] + pitch / 2, hi[d], pitch) for d in range(3)]
    p = np.stack([g.ravel(order="F") for g in np.meshgrid(*ax, indexing="ij")], axis=1)
    x = (p - m.origin) / m.h
    cell = np.floor(x).astype(np.int64)
    order = np.argsort(-(x - cell), axis=1, kind="stable")
    f = -np.sort(-(x - cell), axis=1)
    corner = np.repeat(cell[:, None, :], 4, axis=1)
    for step in range(3):
        corner[np.arange(len(p)), step + 1:, order[:, step]] += 1
    dims = m.lattice.max(0) + 2
    ids = np.full(dims, -1, dtype=np.int64)
    ids[tuple(m.lattice.T)] = np.arange(m.nn)
    inside = ((corner >= 0) & (corner < dims)).all((1, 2))
    node = np.where(inside[:, None], ids[tuple(np.moveaxis(np.clip(corner, 0, dims - 1), 2, 0))], -1)
    w = np.stack([1 - f[:, 0], f[:, 0] - f[:, 1], f[:, 1] - f[:, 2], f[:, 2]], axis=1)
    keep = (node >= 0).all(1)
    rows = np.repeat(np.arange(int(keep.sum())), 4)
    return sp.csr_matrix((w[keep].ravel(), (rows, node[keep].ravel())), shape=(int(keep.sum()), m.nn))


def _fem_args(case):
    return case["shape"], case["size"], case["h"]


# ------------------------------------------------------------- seeded inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _properties(m, gen):
    """Smooth absorption (20 % contrast) and scattering maps over the nodes."""
    x = torch.as_tensor(m.node, device="cuda")
    field = torch.zeros(m.nn, dtype=torch.float64, device="cuda")
    for _ in range(12):
        k = torch.randn(3, generator=gen, dtype=torch.float64, device="cuda") / 8.0
        ph = 2 * math.pi * torch.rand(1, generator=gen, dtype=torch.float64, device="cuda")
        field += torch.cos(x @ k + ph)
    field /= math.sqrt(6.0)
    mua = 0.01 * torch.clamp(1.0 + 0.2 * field, min=0.3)
    return mua, 1.0 + 0.05 * torch.cos(x[:, 0] / 9.0 + field)


def _frequencies(nf):
    return torch.arange(nf, dtype=torch.float64, device="cuda") * (2 * math.pi / T_AXIS[-1])


def _series(x, f):
    """Fourier-series coefficients of signals on the time axis."""
    t = torch.as_tensor(T_AXIS, device="cuda")
    return (x.to(torch.complex128) @ torch.exp(-1j * t[:, None] * f[None, :])) * (T_AXIS[1] / T_AXIS[-1])


def _gates(ng, nf):
    """Fourier coefficients of ng Gaussian gates of 500 ps."""
    t = torch.as_tensor(T_AXIS, device="cuda")
    centre = 0.5e-9 + torch.arange(ng, dtype=torch.float64, device="cuda") * (5e-9 / ng)
    sd = 500e-12 / 2.3548200450309493
    return _series(torch.exp(-((t[None] - centre[:, None]) ** 2) / (2 * sd * sd)), _frequencies(nf)).contiguous()


def _source_spectrum(nf):
    p = torch.as_tensor(workloads.gaussian_pulse(T_AXIS), device="cuda")
    return _series((p * (1e3 / p.mean()))[None], _frequencies(nf))[0].contiguous()


def _fields(m, pos, fpsf, gen):
    """Fluence [nf][nn][n] of point sources: the Green's function of a uniform diffusive medium whose
    absorption the seed sets, with a 2 % ripple over the nodes."""
    x = torch.as_tensor(m.node, device="cuda")
    n, nf = len(pos), fpsf.numel()
    mua = 0.008 + 0.004 * torch.rand(1, generator=gen, dtype=torch.float64, device="cuda")
    d = 1.0 / (3.0 * (mua + 1.0))
    kap = torch.sqrt((mua + 1j * _frequencies(nf) / C_MEDIUM) / d)
    ripple = 1.0 + 0.02 * torch.randn(m.nn, n, generator=gen, dtype=torch.float64, device="cuda")
    r = torch.cdist(x, torch.as_tensor(pos * 0.97, device="cuda")).clamp(min=0.5)
    out = torch.empty((nf, m.nn, n), dtype=torch.complex128, device="cuda")
    for k in range(nf):
        out[k] = fpsf[k] * torch.exp(-kap[k] * r) / (4 * math.pi * d * r) * ripple
    return out


def _sensitivity(case, seed):
    m = _tetmesh(*_fem_args(case))
    gen = _gen(seed)
    ns, nd, nf = case["ns"], case["nd"], case["nf"]
    fpsf = _source_spectrum(nf)
    s = dict(P=_voxels(*_fem_args(case), case["pitch"]) if case["pitch"] else None, fpsf=fpsf,
             phi=_fields(m, _ring(ns, case["shape"], case["size"], 0.0), fpsf, gen),
             phiA=_fields(m, _ring(nd, case["shape"], case["size"], 0.1), fpsf, gen),
             link=torch.as_tensor(workloads.all_pairs(ns, nd).astype(np.int32), device="cuda"))
    nv = s["P"].shape[0] if case["pitch"] else m.nn
    s["w"] = case["pitch"] ** 3 * torch.ones(nv, dtype=torch.float64, device="cuda") if case["pitch"] else \
        case["h"] ** 3 * (0.5 + torch.rand(nv, generator=gen, dtype=torch.float64, device="cuda"))
    if case["kind"] != "jac_fd":
        s["gate"] = _gates(case["ng"], nf)
        shape = (ns * nd, case["ng"])
        s["data"] = torch.exp(3.0 * torch.randn(shape, generator=gen, dtype=torch.float64, device="cuda")) \
            if case["rytov"] else None
        s["g"] = torch.randn(shape, generator=gen, dtype=torch.float64, device="cuda")
    return s


def _lm_inputs(case, seed):
    """A smooth sensitivity matrix with the spread of a Rytov Jacobian, and log-data residuals."""
    gen = _gen(seed)
    nv, nm = case["nv"], case["nm"]
    v = 60 * torch.rand(nv, 3, generator=gen, device="cuda")
    pos = 60 * torch.rand(nm, 2, 3, generator=gen, device="cuda")
    Jt = torch.empty((nv, nm), dtype=torch.float32, device="cuda")
    for a in range(0, nv, 2048):
        q = v[a:a + 2048]
        rs, rd = torch.cdist(q, pos[:, 0]), torch.cdist(q, pos[:, 1])
        Jt[a:a + 2048] = -torch.exp(-0.17 * (rs + rd - (pos[:, 0] - pos[:, 1]).norm(dim=1))) / (1 + rs * rd)
    y = 0.05 * torch.randn(nm, generator=gen, dtype=torch.float64, device="cuda")
    w = None
    if case["weighted"]:
        w = torch.exp(torch.randn(nm, generator=gen, dtype=torch.float64, device="cuda"))
        w /= w.mean()
    return Jt, y, w


def _batch_parts(case):
    """(shape, size, h, ns, nd, nf) of each mesh of a batch: sizes grow, counts shrink and grow again."""
    parts, size = [], case["size"]
    for i in range(case["count"]):
        parts.append((("cylinder", "ellipsoid")[i % 2], round(size * (1.0, 1.35)[i % 2], 2), case["h"],
                      case["ns"] + 3 * (i % 3), case["ns"] + 2, case["nf"] + 5 * (i % 2)))
        size *= case["growth"]
    return parts


# --------------------------------------------------------------- prepare, run
def prepare(case, seed):
    kind = case["kind"]
    if kind == "lm":
        return dict(case=case, inputs=_lm_inputs(case, seed))
    if kind == "batch":
        gen = _gen(seed)
        parts = _batch_parts(case)
        meshes = [_dmesh(*p) for p in parts]
        gates = [_gates(case["ng"], p[5]) for p in parts]
        up = [torch.randn((p[3] * p[4], case["ng"]), generator=gen, dtype=torch.float64, device="cuda")
              for p in parts]
        return dict(case=case, meshes=meshes, props=[_properties(_tetmesh(*p[:3]), gen) for p in parts],
                    gates=gates, up=up,
                    batch=UnevenBatch(meshes, budget_bytes=16 << 30, streams=4, precision="mixed", tol=case["tol"],
                                      gates=gates, upstream=up))
    if kind in ("forward", "gradient"):
        mesh = _dmesh(*_fem_args(case), case["ns"], case["nd"], case["nf"])
        gen = _gen(seed)
        mua, musp = _properties(_tetmesh(*_fem_args(case)), gen)
        s = dict(case=case, mesh=mesh, mua=mua, musp=musp, gate=_gates(case.get("ng", 10), case["nf"]),
                 f=_frequencies(case["nf"]), t=torch.as_tensor(T_AXIS, device="cuda"))
        if kind == "gradient":
            s["model"] = TimeGatedForward(mesh, s["gate"], precision=case["precision"], tol=case["tol"])
            s["g"] = torch.randn((case["ns"] * case["nd"], case["ng"]), generator=gen, dtype=torch.float64,
                                 device="cuda")
        else:
            mesh.solver()
        return s
    s = _sensitivity(case, seed)
    m = _tetmesh(*_fem_args(case))
    return dict(s, case=case, basis=api.Basis(s["P"], s["w"], nn=m.nn))


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "forward":
        mesh = s["mesh"]
        mesh.mua, mesh.musp = s["mua"], s["musp"]
        mesh.update_properties()
        phi, data = mesh.flu_solve(precision=case["precision"], tol=case["tol"])
        return dict(phi=phi, data=data, td=api.fc2td(data, s["f"], s["t"]), tg=api.fc2tg(data, s["gate"], NT))
    if kind == "gradient":
        mua, musp = s["mua"].clone().requires_grad_(), s["musp"].clone().requires_grad_()
        y = s["model"](mua, musp)
        gmua, gmusp = torch.autograd.grad(y, (mua, musp), s["g"])
        return dict(y=y.detach(), gmua=gmua, gmusp=gmusp)
    if kind == "jac_tg":
        return api.jacobian_tg(s["basis"], s["phi"], s["phiA"], s["fpsf"], s["link"], s["gate"], NT, s["data"])
    if kind == "jac_vjp":
        return api.jacobian_tg_vjp(s["basis"], s["phi"], s["phiA"], s["fpsf"], s["link"], s["gate"], NT, s["g"],
                                   s["data"])
    if kind == "jac_fd":
        return api.jacobian_complex(s["basis"], s["phi"], s["phiA"], s["fpsf"], s["link"])
    if kind == "lm":
        Jt, y, w = s["inputs"]
        x = torch.empty(case["nv"], dtype=torch.float64, device="cuda")
        ptr = lambda t: None if t is None else ctypes.c_void_p(t.data_ptr())  # noqa: E731
        check(lib.dgp_lm_update(ptr(Jt), case["nv"], case["nm"], ptr(w), ptr(y), case["lam"], ptr(x), 0, None,
                                api.stream_ptr()))
        return x
    for mesh, (mua, musp) in zip(s["meshes"], s["props"]):
        mesh.mua, mesh.musp = mua, musp
        mesh.update_properties()
    return [dict(data=r.data, vjp=r.vjp) for r in s["batch"].run()]


def work(case):
    kind = case["kind"]
    if kind == "lm":
        nv, nm = case["nv"], case["nm"]
        q = min(nv, nm)
        return dict(bytes=4.0 * nv * nm + 8.0 * (2 * nm + nv), flops=1.0 * q * q * max(nv, nm) + q ** 3 / 3)
    if kind == "batch":
        each = [_solve_work(_tetmesh(*p[:3]).nn, p[3] + p[4], p[5]) for p in _batch_parts(case)]
        return {k: sum(e[k] for e in each) for k in ("bytes", "flops")}
    m = _tetmesh(*_fem_args(case))
    ns, nd, nf = case["ns"], case["nd"], case["nf"]
    if kind == "forward":
        return _solve_work(m.nn, ns, nf)
    if kind == "gradient":
        return _solve_work(m.nn, 2 * ns, nf)
    nv = _voxels(*_fem_args(case), case["pitch"]).shape[0] if case["pitch"] else m.nn
    read = 16.0 * nf * min(m.nn, 4 * nv) * (ns + nd) + 8.0 * nv
    if kind == "jac_fd":
        return dict(bytes=read + 16.0 * nv * nf * ns * nd, flops=14.0 * nv * nf * ns * nd)
    if kind == "jac_tg":
        return dict(bytes=read + 4.0 * nv * case["ng"] * ns * nd, flops=nv * nf * ns * (6.0 * case["ng"] +
                                                                                        4.0 * nd * case["ng"]))
    return dict(bytes=read + 8.0 * nv, flops=8.0 * nv * nf * ns * nd)


def _solve_work(nn, ns, nf):
    """The matrices and the fluence once; per unknown, one application of A and one of its diagonal."""
    return dict(bytes=16.0 * nn * ns * nf + 2 * 12.0 * 15 * nn, flops=nn * ns * nf * 8.0 * 16)


# ------------------------------------------------- the same results in 64 bits
@functools.lru_cache(maxsize=4)
def _p1(shape, size, h):
    """Element geometry and sparsity of linear tetrahedra with Robin faces, on the GPU."""
    m = _tetmesh(shape, size, h)
    e = torch.as_tensor(m.elem.astype(np.int64), device="cuda")
    x = torch.as_tensor(m.node, device="cuda")
    b = torch.stack([x[e[:, q]] - x[e[:, 0]] for q in (1, 2, 3)], dim=2)
    vol = torch.linalg.det(b).abs() / 6
    ref = torch.tensor([[-1.0, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]], dtype=torch.float64, device="cuda")
    grad = torch.einsum("eab,ib->eia", torch.linalg.inv(b.transpose(1, 2)), ref)
    flag = torch.as_tensor(m.bnd, device="cuda")[e]
    es, fs = e[flag.sum(1) == 4], e[flag.sum(1) == 3]
    faces = torch.cat([es[:, [0, 1, 2]], es[:, [0, 1, 3]], es[:, [0, 2, 3]], es[:, [1, 2, 3]],
                       fs[flag[flag.sum(1) == 3]].reshape(-1, 3)])
    area = torch.linalg.cross(x[faces[:, 1]] - x[faces[:, 0]], x[faces[:, 2]] - x[faces[:, 0]]).norm(dim=1) / 2
    r0, ct = (0.4 / 2.4) ** 2, abs(math.cos(math.asin(1 / 1.4)))
    robin = (1 - ct ** 2) / (2 * (2 / (1 - r0) - 1 + ct ** 3))
    key = torch.cat([(e[:, :, None] * m.nn + e[:, None, :]).reshape(-1),
                     (faces[:, :, None] * m.nn + faces[:, None, :]).reshape(-1)])
    pairs, slot = torch.unique(key, return_inverse=True)
    eye3, eye4 = (torch.eye(q, dtype=torch.float64, device="cuda") for q in (3, 4))
    face = (robin * area)[:, None, None] * (1 + eye3) / 12
    mass = vol[:, None, None] * (1 + eye4) / 20
    rows, cols = pairs // m.nn, pairs % m.nn
    crow = torch.searchsorted(rows, torch.arange(m.nn + 1, device="cuda"))
    n16 = mass.numel()
    M = torch.zeros(pairs.numel(), dtype=torch.float64, device="cuda").index_add_(0, slot[:n16], mass.reshape(-1))
    return dict(n=m.nn, e=e, vol=vol, gg=torch.einsum("eia,eja->eij", grad, grad), face=face, slot=slot, rows=rows,
                cols=cols, crow=crow, M=M, eye4=eye4)


def _stiffness(g, mua, musp):
    """Values of K on the pattern (differentiable in the properties)."""
    a, kap = mua[g["e"]], (1 / (3 * (mua + musp)))[g["e"]]
    absorb = (1 + g["eye4"]) * (a.sum(1)[:, None, None] + a[:, :, None] + a[:, None, :]) / 120
    ke = g["vol"][:, None, None] * (g["gg"] * kap.mean(1)[:, None, None] + absorb)
    v = torch.cat([ke.reshape(-1), g["face"].reshape(-1)])
    return torch.zeros_like(g["M"]).index_add(0, g["slot"], v)


def _solve(g, K, omega, B, width=512):
    """X[k] = (K + i omega_k M)^-1 B[k] for B [nf][n][ns]: conjugate-orthogonal CG, twice refined."""
    nf, n, ns = B.shape
    Kc, Mc = (torch.sparse_csr_tensor(g["crow"], g["cols"], v, (n, n)) for v in (K, g["M"]))
    at = g["rows"] == g["cols"]
    dK, dM = K[at], g["M"][at]
    X = torch.empty_like(B)
    per = max(1, width // ns)
    for k0 in range(0, nf, per):
        b = B[k0:k0 + per].permute(1, 0, 2).reshape(n, -1)
        om = omega[k0:k0 + per].repeat_interleave(ns)
        pre = 1 / (dK[:, None] + 1j * dM[:, None] * om)

        def apply(z):
            zr = torch.view_as_real(z).reshape(n, -1)
            kz, mz = ((q @ zr).reshape(n, -1, 2) for q in (Kc, Mc))
            return torch.view_as_complex(kz) + 1j * om * torch.view_as_complex(mz)

        x, r, norm = torch.zeros_like(b), b.clone(), b.norm(dim=0).clamp(min=1e-300)
        for _ in range(3):
            d, p, rho, q = torch.zeros_like(b), None, None, r.clone()
            first = (q.norm(dim=0)).clamp(min=1e-300)
            for it in range(2000):
                if it % 8 == 0 and float((q.norm(dim=0) / first).max()) < 1e-9:
                    break
                z = pre * q
                new = (q * z).sum(0)
                p = z if p is None else z + torch.nan_to_num(new / rho) * p
                rho = new
                ap = apply(p)
                a = torch.nan_to_num(rho / (p * ap).sum(0))
                d += a * p
                q -= a * ap
            x += d
            r = b - apply(x)
            if float((r.norm(dim=0) / norm).max()) < 2e-15:
                break
        X[k0:k0 + per] = x.reshape(n, -1, ns).permute(1, 0, 2)
    return X


def _points(mesh, bary):
    """Nodes [n][4] and weights [n][4] of the optodes of a mesh."""
    bary = np.asarray(bary)
    nodes = torch.as_tensor(mesh.elem_host[bary[:, 0].astype(np.int64)], device="cuda")
    return nodes, torch.as_tensor(np.ascontiguousarray(bary[:, 1:5]), device="cuda")


def _rhs(mesh, bary, fpsf):
    nodes, w = _points(mesh, bary)
    B = torch.zeros((fpsf.numel(), mesh.nn, len(nodes)), dtype=torch.complex128, device="cuda")
    for q in range(4):
        B[:, nodes[:, q], torch.arange(len(nodes), device="cuda")] = fpsf[:, None] * w[:, q]
    return B


def _readout(mesh, phi):
    """Detector data [ns * nd][nf], every source with every detector."""
    nodes, w = _points(mesh, mesh.optode.d_bary)
    at = (phi[:, nodes.reshape(-1)].reshape(phi.shape[0], *nodes.shape, -1) * w[None, :, :, None]).sum(2)
    return at.permute(2, 1, 0).reshape(-1, phi.shape[0])


def _halved(c):
    return torch.cat([0.5 * c[:, :1], c[:, 1:]], dim=1)


def _gated(data, gate):
    return 2 * NT * (_halved(data) @ gate.conj().T).real


def _forward64(mesh, geometry, mua, musp, nf):
    g = _p1(*geometry)
    K = _stiffness(g, mua, musp)
    fpsf = _source_spectrum(nf)
    om = _frequencies(nf) / C_MEDIUM
    return g, K, om, fpsf, _solve(g, K, om, _rhs(mesh, mesh.optode.s_bary, fpsf))


def _project(P, phi):
    """Fields on the basis [nv][nf][n]."""
    if P is None:
        return phi.permute(1, 0, 2)
    Pt = torch.sparse_csr_tensor(torch.as_tensor(P.indptr), torch.as_tensor(P.indices), torch.as_tensor(P.data),
                                 P.shape).to("cuda")
    flat = torch.view_as_real(phi.permute(1, 0, 2).contiguous()).reshape(phi.shape[1], -1)
    return torch.view_as_complex((Pt @ flat).reshape(P.shape[0], phi.shape[0], phi.shape[2], 2))


def _vjp64(P, w, phi, phiA, fpsf, gate, g, data):
    nf, ns, nd = phi.shape[0], phi.shape[2], phiA.shape[2]
    if data is not None:
        g = g / data
    c = -2 * NT / fpsf * torch.where(torch.arange(nf, device="cuda") == 0, 0.5, 1.0)
    h = ((g.to(torch.complex128) @ gate.conj()) * c).T.reshape(nf, ns, nd)
    out = []
    for a in range(0, len(w), 8192):
        sel = P[a:a + 8192] if P is not None else None
        x, y = (_project(sel, f if P is not None else f[:, a:a + 8192]) for f in (phi, phiA))
        out.append(torch.einsum("vks,ksd,vkd->v", x, h, y).real if ns * nd < 4 else
                   (x * torch.einsum("ksd,vkd->vks", h, y)).sum((1, 2)).real)
    return torch.cat(out) * w


def _jacobian64(s, case):
    nf = case["nf"]
    n = case["ns"] * case["nd"]
    step = max(64, int(2.5e8 / (nf * n)))
    out = []
    for a in range(0, len(s["w"]), step):
        x, y = (_project(None if s["P"] is None else s["P"][a:a + step],
                         f if s["P"] is not None else f[:, a:a + step]) for f in (s["phi"], s["phiA"]))
        J = -(x[:, :, :, None] * y[:, :, None, :]).reshape(len(x), nf, n) / s["fpsf"][:, None] * \
            s["w"][a:a + step, None, None]
        if case["kind"] == "jac_tg":
            J[:, 0] *= 0.5
            J = torch.view_as_real(J).permute(0, 2, 1, 3).reshape(-1, 2 * nf)
            J = (J @ torch.view_as_real(s["gate"]).reshape(-1, 2 * nf).T).mul_(2 * NT)
            J = J.reshape(len(x), n, -1).transpose(1, 2)
            if s["data"] is not None:
                J = J / s["data"].T
        out.append(J)
    return torch.cat(out)


def _gradient64(case, seed):
    s = prepare(case, seed)
    mesh, ns, nd, nf = s["mesh"], case["ns"], case["nd"], case["nf"]
    g, K, om, fpsf, phi = _forward64(mesh, _fem_args(case), s["mua"], s["musp"], nf)
    c = 2 * NT * _halved(s["g"].to(torch.complex128) @ s["gate"].conj()).reshape(ns, nd, nf)
    nodes, w = _points(mesh, mesh.optode.d_bary)
    B = torch.zeros_like(phi)
    for q in range(4):
        B.index_add_(1, nodes[:, q], (c * w[None, :, q, None]).permute(2, 1, 0).contiguous())
    lam = _solve(g, K, om, B)
    S = torch.zeros_like(g["M"])
    for k in range(nf):
        S += (lam[k][g["rows"]] * phi[k][g["cols"]]).sum(1).real
    mua, musp = s["mua"].clone().requires_grad_(), s["musp"].clone().requires_grad_()
    gmua, gmusp = torch.autograd.grad(-(_stiffness(g, mua, musp) * S).sum(), (mua, musp))
    return dict(y=_gated(_readout(mesh, phi), s["gate"]), gmua=gmua, gmusp=gmusp)


def exact(case, seed):
    kind = case["kind"]
    if kind == "forward":
        s = prepare(case, seed)
        phi = _forward64(s["mesh"], _fem_args(case), s["mua"], s["musp"], case["nf"])[-1]
        data = _readout(s["mesh"], phi)
        td = 2 * (_halved(data) @ torch.exp(1j * s["f"][:, None] * s["t"][None])).real
        return dict(phi=phi, data=data, td=td, tg=_gated(data, s["gate"]))
    if kind == "gradient":
        return _gradient64(case, seed)
    if kind in ("jac_tg", "jac_fd"):
        return _jacobian64(_sensitivity(case, seed), case)
    if kind == "jac_vjp":
        s = _sensitivity(case, seed)
        return _vjp64(s["P"], s["w"], s["phi"], s["phiA"], s["fpsf"], s["gate"], s["g"], s["data"])
    if kind == "lm":
        Jt, y, w = _lm_inputs(case, seed)
        J = Jt.double()
        if w is not None:
            J *= torch.sqrt(w)
            y = torch.sqrt(w) * y
        mu = case["lam"] * (J * J).sum(1).max()
        wide = J.shape[0] > J.shape[1]
        H = J.T @ J if wide else J @ J.T
        H.diagonal().add_(mu)
        L = torch.linalg.cholesky(H)
        b = y if wide else J @ y
        z = torch.cholesky_solve(b[:, None], L)[:, 0]
        return J @ z if wide else z
    s = prepare(case, seed)
    out = []
    for p, mesh, (mua, musp), gate, up in zip(_batch_parts(case), s["meshes"], s["props"], s["gates"], s["up"]):
        g, K, om, fpsf, phi = _forward64(mesh, p[:3], mua, musp, p[5])
        phiA = _solve(g, K, om, _rhs(mesh, mesh.optode.d_bary, fpsf))
        lump = torch.zeros(g["n"], dtype=torch.float64, device="cuda").index_add_(0, g["rows"], g["M"])
        out.append(dict(data=_readout(mesh, phi), vjp=_vjp64(None, lump, phi, phiA, fpsf, gate, up, None)))
    return out
