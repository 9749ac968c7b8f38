"""The fused COCG solve (three sweeps per iteration, harmonics solved in levels with initial
guesses combined from earlier levels) against sparse-direct solutions.

Tolerance: a column's FP64 relative residual is below tol = 1e-11 on return; the matrices' condition
number here is below 1e4, so the fluence is within 1e-6 per right-hand side (the bar of the mixed
solves) with orders to spare."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

C_MED = 2.99792458e11 / 1.4
DFC = 2 * np.pi / 10e-9 / C_MED


@pytest.fixture(scope="module")
def case():
    import torch
    from dogpup_b200 import api, meshgen
    from oracle import fem
    m = meshgen.cylinder_mesh(10.0, 16.0, 1.5, jitter=0.2, seed=1)
    rng = np.random.default_rng(0)
    mua, musp = 0.01 * (1 + 0.3 * rng.random(m.nn)), 1 + 0.2 * rng.random(m.nn)
    K, M = fem.gen_fwdmat(m.node, m.elem, fem.prepare_mesh(m.node, m.elem, 1.4), mua, musp)
    f = api.Fem(torch.as_tensor(m.node), torch.as_tensor(m.elem), 1.4)
    Kd, Md = f.assemble(torch.as_tensor(mua), torch.as_tensor(musp))
    return dict(m=m, K=K, M=M, fem=f, Kd=Kd, Md=Md)


def _solve(case, ns, harm, fpsf, seed=3, **kw):
    import torch
    from dogpup_b200 import api
    m = case["m"]
    rng = np.random.default_rng(seed)
    nodes = m.elem[rng.choice(m.ne, ns, replace=False)].astype(np.int32)
    w = rng.random((ns, 4))
    w /= w.sum(1, keepdims=True)
    S = api.Solver(case["fem"].rowptr, case["fem"].col, case["Kd"], case["Md"], DFC, len(harm), ns, harmonics=harm)
    status = torch.full((len(harm) * ns,), -1, dtype=torch.int32, device="cuda")
    X, rep = S.solve_sources(torch.as_tensor(nodes, device="cuda"), torch.as_tensor(w, device="cuda"),
                             torch.as_tensor(np.asarray(fpsf, dtype=complex), device="cuda"),
                             api.make_opts(precision="mixed", **{"tol": 1e-11, **kw}), status=status)
    return nodes, w, X.cpu().numpy(), rep, status.cpu().numpy().reshape(len(harm), ns)


def _check(case, nodes, w, X, harm, fpsf, which):
    import scipy.sparse.linalg as sla
    n, ns = case["K"].shape[0], len(w)
    B = np.zeros((n, ns))
    for s in range(ns):
        B[nodes[s], s] = w[s]
    for j in which:
        x = sla.splu((case["K"] + 1j * harm[j] * DFC * case["M"]).tocsc()).solve(B.astype(complex)) * fpsf[j]
        norm = np.linalg.norm(x, axis=0)
        err = np.linalg.norm(X[j] - x, axis=0)
        assert (err <= 1e-6 * np.where(norm > 0, norm, 1.0)).all(), (j, err.max())


@pytest.mark.parametrize("ns", [1, 3, 5, 8, 11, 16, 23, 33, 47, 128])
def test_source_counts(case, ns):
    """Lane widths and padded columns: 4 to 128 columns, rows of 2 to 32 lanes, idle lanes included."""
    harm, fpsf = [0, 3, 17], np.exp(-0.3j * np.arange(3))
    nodes, w, X, rep, st = _solve(case, ns, harm, fpsf)
    assert (st == 0).all() and rep.max_rel_residual < 1e-11
    _check(case, nodes, w, X, harm, fpsf, range(3))


@pytest.mark.parametrize("nf", [16, 17, 40])
def test_levels(case, nf):
    """Enough columns for several levels; a spectrum over 12 decades."""
    harm, fpsf = list(range(nf)), 10.0 ** (-12 * np.arange(nf) / nf) * np.exp(0.4j * np.arange(nf))
    nodes, w, X, rep, st = _solve(case, 66, harm, fpsf)
    assert (st == 0).all() and rep.max_rel_residual < 1e-11
    _check(case, nodes, w, X, harm, fpsf, [0, 1, 2, nf // 2, nf - 2, nf - 1])


def test_levels_on_scattered_harmonics_with_silent_ones(case):
    """Unordered, widely spaced and repeated harmonics, some without source strength: a silent harmonic
    gives zero and offers nothing to the others' guesses."""
    harm = [90, 0, 7, 7, 31, 2, 64, 5, 120, 1, 13, 44, 3, 19, 77, 200, 8, 26, 55, 4]
    fpsf = np.exp(-0.1j * np.arange(len(harm)))
    fpsf[[1, 6, 15]] = 0.0
    nodes, w, X, rep, st = _solve(case, 70, harm, fpsf)
    assert (st == 0).all() and rep.max_rel_residual < 1e-11
    assert np.abs(X[[1, 6, 15]]).max() == 0.0
    _check(case, nodes, w, X, harm, fpsf, range(len(harm)))


def test_level_count_does_not_change_maxit(case):
    """maxit bounds every column's iterations in each level."""
    nodes, w, X, rep, st = _solve(case, 66, list(range(20)), np.ones(20), maxit=5, check_every=1, tol=1e-13)
    assert rep.iterations == 5 and (st == 1).any() and np.isfinite(X).all()


def test_nonfinite_source_keeps_the_others(case):
    import torch
    from dogpup_b200 import api
    m, ns, harm = case["m"], 65, list(range(16))
    rng = np.random.default_rng(8)
    nodes = m.elem[rng.choice(m.ne, ns, replace=False)].astype(np.int32)
    w = rng.random((ns, 4))
    w[7, 2] = np.nan
    S = api.Solver(case["fem"].rowptr, case["fem"].col, case["Kd"], case["Md"], DFC, 16, ns)
    status = torch.full((16 * ns,), -1, dtype=torch.int32, device="cuda")
    X, rep = S.solve_sources(torch.as_tensor(nodes, device="cuda"), torch.as_tensor(w, device="cuda"),
                             torch.ones(16, dtype=torch.complex128, device="cuda"),
                             api.make_opts(precision="mixed", tol=1e-11), status=status)
    st = status.cpu().numpy().reshape(16, ns)
    keep = np.arange(ns) != 7
    assert (st[:, 7] == 4).all() and (st[:, keep] == 0).all() and rep.n_not_converged == 16
    _check(case, nodes[keep], w[keep], X.cpu().numpy()[:, :, keep], harm, np.ones(16), [0, 5, 15])


def test_forward_and_adjoint_solves_share_a_plan_without_allocating(case):
    """Point-source and dense solves in turn on one plan, as a gradient step makes them: after one of each
    the plan holds all it needs, and the results stay the same."""
    import torch
    from dogpup_b200 import api
    from dogpup_b200._lib import lib
    m, ns, nf = case["m"], 66, 20
    rng = np.random.default_rng(4)
    nodes = m.elem[rng.choice(m.ne, ns, replace=False)].astype(np.int32)
    w = np.full((ns, 4), 0.25)
    S = api.Solver(case["fem"].rowptr, case["fem"].col, case["Kd"], case["Md"], DFC, nf, ns)
    src = [torch.as_tensor(a, device="cuda") for a in (nodes, w, np.ones(nf, dtype=complex))]
    B = torch.zeros((nf, m.nn, ns), dtype=torch.complex128, device="cuda")
    for s in range(ns):
        B[:, torch.as_tensor(nodes[s].astype(np.int64), device="cuda"), s] = 0.25
    opts = api.make_opts(precision="mixed", tol=1e-11)
    steps = []
    for _ in range(3):
        a0 = lib.dgp_device_allocations()
        X, r = S.solve_sources(*src, opts)
        Y, q = S.solve(B, opts)
        assert r.n_not_converged == 0 and q.n_not_converged == 0
        _check(case, nodes, w, X.cpu().numpy(), range(nf), np.ones(nf), [0, 7, 19])
        _check(case, nodes, w, Y.cpu().numpy(), range(nf), np.ones(nf), [0, 7, 19])
        steps.append(lib.dgp_device_allocations() - a0)
    assert steps[0] > 0 and steps[1:] == [0, 0]
